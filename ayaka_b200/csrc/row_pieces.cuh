// Rows of fp32 numbers in pieces of four entries, in registers: kernels that norm rows or join them to
// the residual stream are bound by memory, and with 4-byte accesses a row's loads and stores do not
// cover the trip. A thread holds P pieces, blockDim.x apart: 2, or ROW_PIECES for rows of more than 4,096
// entries (held for all rows, the registers of ROW_PIECES leave half the warps: norm_add over 4,096 rows
// of 4,096 with a copy and the next norm 85 microseconds where this takes 53).
#pragma once

#include "common.cuh"

namespace ayk {

constexpr int ROW_PIECES = 4;
__device__ __forceinline__ float4 row_piece(const float* row, int piece, int pieces) {
  return piece < pieces ? reinterpret_cast<const float4*>(row)[piece]
                        : make_float4(0.f, 0.f, 0.f, 0.f);
}
__device__ __forceinline__ float4 offset_piece(const float* w, float offset, int piece, int pieces) {
  float4 v = row_piece(w, piece, pieces);
  v.x += offset;
  v.y += offset;
  v.z += offset;
  v.w += offset;
  return v;
}
__device__ __forceinline__ float square_sum(const float4& v) {
  return fmaf(v.x, v.x, v.y * v.y) + fmaf(v.z, v.z, v.w * v.w);
}
__device__ __forceinline__ void put_piece(float* row, int piece, const float4& v) {
  reinterpret_cast<float4*>(row)[piece] = v;
}
__device__ __forceinline__ void put_piece(__nv_bfloat16* row, int piece, const float4& v) {
  const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
  reinterpret_cast<uint2*>(row)[piece] = make_uint2(*reinterpret_cast<const uint32_t*>(&a),
                                                    *reinterpret_cast<const uint32_t*>(&b));
}
// Four entries of the compute type as fp32.
__device__ __forceinline__ float4 load_piece(const float* row, int piece) {
  return reinterpret_cast<const float4*>(row)[piece];
}
__device__ __forceinline__ float4 load_piece(const __nv_bfloat16* row, int piece) {
  const uint2 raw = reinterpret_cast<const uint2*>(row)[piece];
  return make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u),
                     __uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xffff0000u));
}
// A vector that every row is multiplied with: fetched ahead of the wait for the kernel before (a few
// rows' time is a chain of trips to memory) where the registers allow it, else where it is used. A null
// one is `without`.
template <int P> struct RowWeights {
  static constexpr bool AHEAD = P <= 2;
  float4 held[AHEAD ? P : 1];
  const float* from;
  int pieces;
  float without;
  __device__ __forceinline__ RowWeights(const float* w, int pieces_, float without_)
      : from(w), pieces(pieces_), without(without_) {
    if (AHEAD) {
#pragma unroll
      for (int i = 0; i < P; ++i) held[AHEAD ? i : 0] = fetch(i);
    }
  }
  __device__ __forceinline__ float4 fetch(int i) const {
    return from != nullptr ? row_piece(from, threadIdx.x + i * blockDim.x, pieces)
                           : make_float4(without, without, without, without);
  }
  __device__ __forceinline__ float4 piece(int i) const {
    if constexpr (AHEAD) {
      return held[i];
    } else {
      return fetch(i);
    }
  }
};
// out = the root-mean-square norm of the row held in `v` (the norm in front of the next sublayer);
// s2: this thread's sum of squares.
template <int P, typename TOut>
__device__ __forceinline__ void next_norm(const float4 (&v)[P], float s2, float* scratch, int width,
                                          const RowWeights<P>& weight, float offset, float eps,
                                          TOut* out) {
  const int pieces = width / 4;
  const float inv = 1.f / sqrtf(block_sum(s2, scratch) / (float)width + eps);
#pragma unroll
  for (int i = 0; i < P; ++i) {
    const int c = threadIdx.x + i * blockDim.x;
    if (c < pieces) {
      float4 w = weight.piece(i);
      w.x += offset;
      w.y += offset;
      w.z += offset;
      w.w += offset;
      put_piece(out, c, make_float4(v[i].x * inv * w.x, v[i].y * inv * w.y, v[i].z * inv * w.z,
                                    v[i].w * inv * w.w));
    }
  }
}
// Whether rows of `width` at `p`, `ld` entries of `bytes` apart, are whole pieces (a null p is).
inline bool row_takes(const void* p, long long ld, int width, int bytes) {
  return p == nullptr || (width % 4 == 0 && ld % 4 == 0 && (uintptr_t)p % (4 * bytes) == 0);
}
// Threads of a CTA that holds a row, by the width alone (a row's sums do not depend on the step): two
// pieces a thread, which a decode step's few rows need (four were 0.5 % of a step slower), up to
// ROW_PIECES where that is more than 512 threads. 0: the row does not fit.
inline int row_threads(int width) {
  const int pieces = width / 4, two = (pieces + 1) / 2, most = (pieces + ROW_PIECES - 1) / ROW_PIECES;
  const int want = two <= 512 ? two : most;
  return want <= 64 ? 64 : (want <= 512 ? (want + 31) / 32 * 32 : 0);
}
// Whether two pieces a thread hold a row.
inline bool row_in_two(int width, int threads) { return width / 4 <= 2 * threads; }

}  // namespace ayk
