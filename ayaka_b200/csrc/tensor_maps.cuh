// Tensor maps of row-major matrices, encoded once each.
#pragma once

#include <mutex>
#include <unordered_map>

#include "tc_common.cuh"

namespace ayk {

// Tensor maps are cached by what they describe: weights are static and activations live in
// persistent buffers, so a serving process encodes each map once.
struct MapKey {
  const void* base;
  uint64_t rows, cols, ld;
  uint32_t box_rows, elem_bytes;
  bool operator==(const MapKey& o) const {
    return base == o.base && rows == o.rows && cols == o.cols && ld == o.ld &&
           box_rows == o.box_rows && elem_bytes == o.elem_bytes;
  }
};
struct MapKeyHash {
  size_t operator()(const MapKey& k) const {
    size_t h = (size_t)k.base;
    h = h * 1000003u ^ k.rows;
    h = h * 1000003u ^ k.cols;
    h = h * 1000003u ^ k.ld;
    h = h * 1000003u ^ k.box_rows;
    h = h * 1000003u ^ k.elem_bytes;
    return h;
  }
};

static int cached_map(const void* base, uint64_t rows, uint64_t cols, uint64_t ld,
                      uint32_t box_rows, CUtensorMap* out, int elem_bytes = 2) {
  static std::mutex mu;
  static std::unordered_map<MapKey, CUtensorMap, MapKeyHash> cache;
  std::lock_guard<std::mutex> lock(mu);
  const MapKey key{base, rows, cols, ld, box_rows, (uint32_t)elem_bytes};
  auto it = cache.find(key);
  if (it == cache.end()) {
    CUtensorMap map;
    const int r = make_map_128b(&map, base, rows, cols, ld, box_rows, elem_bytes);
    if (r != AYK_OK) return r;
    if (cache.size() > 4096) cache.clear();
    it = cache.emplace(key, map).first;
  }
  *out = it->second;
  return AYK_OK;
}

}  // namespace ayk
