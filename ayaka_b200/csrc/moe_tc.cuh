// The experts' grouped products of many rows on the 5th-generation tensor cores (bfloat16).
//
// Bound by tcgen05 throughput once an expert gets a few hundred pairs, by reading every expert's
// matrices once below that. A persistent CTA per SM walks tiles of 128 pairs of one expert x 256
// columns, two accumulators in tensor memory, so that a tile's epilogue runs under the next
// tile's main loop. Six warps: warp 0 fills the ring of four stages, warp 1's elected thread
// issues the MMAs, warps 2-5 are the epilogue.
//   PHASE 0: a tile's 128 rows are contiguous in a copy of the input grouped by expert
//            (moe_group_kernel). The 256 columns are 128 gate and the 128 up columns that go with
//            them, so the unit is formed in the epilogue's registers from both in fp32; an expert
//            without a gate has 256 up columns. Gathering the rows by TMA instead (tile::gather4,
//            32 a stage) took 357 microseconds where this takes 152 with its copy (8,192 pairs,
//            2,048 x 2 x 2,048): four rows an instruction do not keep up with the MMAs.
//   PHASE 1: rows are the tile's contiguous places of PHASE 0's output; a warp's 32 x 32 piece is
//            turned through shared memory so that eight lanes store 128 contiguous bytes of a
//            pair's row (one lane a row touches 32 lines per instruction).
// Tiles run columns first: the tiles that run at one time share few experts' matrices, which
// then come from DRAM once. Results do not depend on a pair's place: k runs upward in blocks of
// 64 for every tile.
//
// Measured on a B200, against mma.sync tiles of 128 x 64 (both products of a layer, device time):
// 8,192 pairs, 16 gated experts, 2,048 x 2,048: 965 -> 235 microseconds with the grouping (205 GFLOP,
// 870 TFLOP/s; 400 MB of matrices are 62); 8,192 pairs, 1,024 x 1,024 without a gate: 234 -> 71. The
// tensor pipe is active for 71 % of the first product's time and 62 % of the second's.
#pragma once

#include "tc_common.cuh"

namespace ayk {

constexpr int MT_ROWS = 128, MT_COLS = 256, MT_K = 64, MT_STAGES = 4;
constexpr int MT_A_BYTES = MT_ROWS * MT_K * 2;
constexpr int MT_HALF_BYTES = MT_COLS / 2 * MT_K * 2;  // a box of 128 weight rows
constexpr int MT_STAGE_BYTES = MT_A_BYTES + 2 * MT_HALF_BYTES;
constexpr int MT_WARP_BYTES = 32 * 128;  // an epilogue warp's box: 32 rows x 128 bytes
constexpr int MT_EPI_OFFSET = MT_STAGES * MT_STAGE_BYTES;
constexpr int MT_BAR_OFFSET = MT_EPI_OFFSET + 4 * MT_WARP_BYTES;
// full, empty per stage; acc_full, acc_empty per accumulator; tensor-memory slot, failure flag
constexpr int MT_DYNAMIC = MT_BAR_OFFSET + (2 * MT_STAGES + 4) * 8 + 16 + 1024;

struct MoeUnit {
  float limit, alpha, shift;
  int single;
};

// The input's rows grouped by expert, without gaps: pair `sorted[place]`'s row goes to row
// tile_first[tile] + (place - the tile's first) of `to`. A warp per place copies 16 bytes a lane;
// bound by writing pairs x width x 2 bytes (the rows come from L2).
__global__ void __launch_bounds__(256)
moe_group_kernel(const __nv_bfloat16* __restrict__ hidden, int ld_hidden,
                 const int* __restrict__ sorted, const int* __restrict__ tile_expert,
                 const int* __restrict__ tile_first, int top, int width,
                 __nv_bfloat16* __restrict__ to, long long ld_to) {
  pdl_launch_dependents();
  const int tile = blockIdx.x, r = blockIdx.y * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  pdl_wait_for(hidden, sorted, tile_expert, tile_first, to);
  if (tile_expert[tile] < 0) return;
  const int pair = sorted[(size_t)tile * MT_ROWS + r];
  if (pair < 0) return;
  const uint4* src = reinterpret_cast<const uint4*>(hidden + (size_t)(pair / top) * ld_hidden);
  uint4* dst = reinterpret_cast<uint4*>(to + (size_t)(tile_first[tile] + r) * ld_to);
#pragma unroll 4
  for (int c = lane; c < width / 8; c += 32) dst[c] = src[c];
}

// map_a: PHASE 0 the grouped input, PHASE 1 the places (boxes of 128 rows); map_w: the experts'
// matrices (boxes of 128 rows); map_y: PHASE 0's output (boxes of 32 rows).
template <int PHASE>
__global__ void __launch_bounds__(192)
moe_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
              const __grid_constant__ CUtensorMap map_y, const int* __restrict__ sorted,
              const int* __restrict__ tile_expert, const int* __restrict__ tile_first,
              int max_tiles, int K, int N, MoeUnit unit, float* __restrict__ out, int ld_out,
              int* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + MT_BAR_OFFSET);
  uint64_t* empty = full + MT_STAGES;
  uint64_t* acc_full = empty + MT_STAGES;
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool gated = PHASE == 0 && !unit.single;
  const int tile_cols = gated ? MT_COLS / 2 : MT_COLS;  // output columns of a tile
  const int tiles_n = (N + tile_cols - 1) / tile_cols;
  const int num_kb = (K + MT_K - 1) / MT_K;
  constexpr uint32_t TMEM_COLS = 2 * MT_COLS;

  if (threadIdx.x == 0) {
    for (int s = 0; s < MT_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 4);
    }
    *failed = 0;
    mbar_fence_init();
    tma_prefetch_map(&map_a);
    tma_prefetch_map(&map_w);
  }
  if (warp == 0) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();
  pdl_wait_for(sorted, tile_expert, tile_first);

  // this CTA's tile t: its row tile, its expert (-1: there is none, nor behind it) and column
  const int all = max_tiles * tiles_n;
  auto expert_of = [&](int t) { return t < all ? tile_expert[t / tiles_n] : -1; };

  if (warp == 0 && lane == 0) {
    // ---- producer
    int it = 0;
    bool ok = true;
    for (int t = blockIdx.x; ok && *failed == 0; t += gridDim.x) {
      const int e = expert_of(t);
      if (e < 0) break;
      const int m = t / tiles_n, n0 = (t - m * tiles_n) * tile_cols;
      // (a grouped tile's rows run on into the next expert's, or end with the tensor: their
      // results are never used)
      const int m0 = PHASE == 0 ? tile_first[m] : m * MT_ROWS;
      const int w_row = e * (gated ? 2 : 1) * N + n0;
      const int w_row2 = w_row + (gated ? N : MT_COLS / 2);
      for (int kb = 0; kb < num_kb; ++kb, ++it) {
        const int s = it % MT_STAGES;
        uint8_t* a_tile = smem + s * MT_STAGE_BYTES;
        if (it >= MT_STAGES && !mbar_wait(&empty[s], ((it / MT_STAGES) & 1) ^ 1)) {
          *failed = 1;
          ok = false;
          break;
        }
        mbar_expect_tx(&full[s], MT_STAGE_BYTES);
        tma_load_2d(a_tile, &map_a, &full[s], kb * MT_K, m0);
        tma_load_2d(a_tile + MT_A_BYTES, &map_w, &full[s], kb * MT_K, w_row);
        tma_load_2d(a_tile + MT_A_BYTES + MT_HALF_BYTES, &map_w, &full[s], kb * MT_K, w_row2);
      }
    }
    if (*failed != 0) {  // copies in flight land in this CTA's memory: wait, with a limit
      for (int i = it > MT_STAGES ? it - MT_STAGES : 0; i < it; ++i) {
        mbar_wait(&full[i % MT_STAGES], (i / MT_STAGES) & 1);
      }
    }
  } else if (warp == 1 && lane == 0) {
    // ---- MMA issuer
    constexpr uint32_t idesc = umma_idesc_bf16(MT_ROWS, MT_COLS);
    int it = 0, local = 0;
    for (int t = blockIdx.x; *failed == 0 && expert_of(t) >= 0; t += gridDim.x, ++local) {
      const int buf = local & 1;
      if (local >= 2 && !mbar_wait(&acc_empty[buf], ((local >> 1) & 1) ^ 1)) {
        *failed = 1;
        break;
      }
      tc_fence_after();
      const uint32_t acc = tmem_base + (uint32_t)(buf * MT_COLS);
      bool ok = true;
      for (int kb = 0; kb < num_kb; ++kb, ++it) {
        const int s = it % MT_STAGES;
        if (!mbar_wait(&full[s], (it / MT_STAGES) & 1)) {
          *failed = 1;
          ok = false;
          break;
        }
        tc_fence_after();
        const uint8_t* a_tile = smem + s * MT_STAGE_BYTES;
#pragma unroll
        for (int k = 0; k < MT_K / 16; ++k) {
          umma_f16(acc, umma_desc_k128(a_tile, k * 32), umma_desc_k128(a_tile + MT_A_BYTES, k * 32),
                   idesc, (kb | k) != 0);
        }
        umma_commit(&empty[s]);
      }
      if (!ok) break;
      umma_commit(&acc_full[buf]);
    }
  } else if (warp >= 2) {
    // ---- epilogue: warp w reads tensor-memory lanes 32 (w % 4) ..
    const int quarter = warp & 3;
    uint8_t* staging = smem + MT_EPI_OFFSET + quarter * MT_WARP_BYTES;
    uint8_t* row = staging + lane * 128;
    const int swz = lane & 7;
    int local = 0;
    for (int t = blockIdx.x; expert_of(t) >= 0; t += gridDim.x, ++local) {
      const int buf = local & 1;
      const int m = t / tiles_n, n0 = (t - m * tiles_n) * tile_cols;
      const int m_warp = m * MT_ROWS + quarter * 32;
      const int pair = PHASE == 1 ? sorted[m_warp + lane] : 0;
      bool have = true;
      if (lane == 0) have = mbar_wait(&acc_full[buf], (local >> 1) & 1);
      have = __shfl_sync(0xffffffffu, have, 0);
      if (!have || *failed != 0) {
        if (lane == 0) *failed = 1;
        break;
      }
      tc_fence_after();
      const uint32_t acc =
          tmem_base + (uint32_t)(buf * MT_COLS) + ((uint32_t)(quarter * 32) << 16);
#pragma unroll 1
      for (int c = 0; c < tile_cols / 32; ++c) {
        const int n = n0 + c * 32;
        if (n >= N) break;
        uint32_t raw[32];
        tmem_ld_32x32(acc + (uint32_t)(c * 32), raw);
        if (PHASE == 0) {
          float v[32];
          if (gated) {
            uint32_t up[32];
            tmem_ld_32x32(acc + (uint32_t)(MT_COLS / 2 + c * 32), up);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              v[j] = expert_unit(__uint_as_float(raw[j]), __uint_as_float(up[j]), unit.limit,
                                 unit.alpha, unit.shift, 0);
            }
          } else {
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = relu_squared(__uint_as_float(raw[j]));
          }
          if ((c & 1) == 0) {  // a box is two chunks of 32 columns
            if (lane == 0) bulk_wait_read_all();
            __syncwarp();
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint32_t packed[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const __nv_bfloat162 h =
                  __floats2bfloat162_rn(v[q * 8 + 2 * i], v[q * 8 + 2 * i + 1]);
              packed[i] = *reinterpret_cast<const uint32_t*>(&h);
            }
            *reinterpret_cast<uint4*>(row + ((((c & 1) * 4 + q) ^ swz) << 4)) =
                make_uint4(packed[0], packed[1], packed[2], packed[3]);
          }
          if ((c & 1) == 1 || n + 32 >= N) {
            fence_proxy_async_shared();
            __syncwarp();
            if (lane == 0) {
              tma_store_2d(&map_y, staging, n0 + (c & ~1) * 32, m_warp);
              bulk_commit_group();
            }
          }
        } else {
          tmem_ld_wait();
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            *reinterpret_cast<uint4*>(row + ((q ^ swz) << 4)) =
                make_uint4(raw[q * 4], raw[q * 4 + 1], raw[q * 4 + 2], raw[q * 4 + 3]);
          }
          __syncwarp();
          const int piece = lane & 7;
          const bool in = n + piece * 4 < N;  // (N is a multiple of 8)
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int r = i * 4 + (lane >> 3);
            const int to = __shfl_sync(0xffffffffu, pair, r);
            const float4 v =
                *reinterpret_cast<const float4*>(staging + r * 128 + ((piece ^ (r & 7)) << 4));
            if (to >= 0 && in) {
              *reinterpret_cast<float4*>(out + (size_t)to * ld_out + n + piece * 4) = v;
            }
          }
          __syncwarp();
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
    }
    if (PHASE == 0 && lane == 0) bulk_wait_all();
  }

  tc_fence_before();
  __syncthreads();
  if (*failed != 0 && threadIdx.x == 0) atomicExch(status, AYK_WAIT_TIMEOUT);
  if (warp == 0) {
    __syncwarp();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// Whether the tensor-core products take these operands: TMA reads and the vector stores need
// 16-byte aligned bases and rows.
inline bool moe_tc_takes(const void* hidden, int ld_hidden, const void* w_in, const void* w_out,
                         int width, int ff, const void* y, int ld_y, const float* pair_out,
                         int ld_out) {
  const auto aligned = [](const void* p) { return ((uintptr_t)p % 16) == 0; };
  return width % 8 == 0 && ff % 8 == 0 && ld_hidden % 8 == 0 && ld_y % 8 == 0 &&
         ld_out % 4 == 0 && aligned(hidden) && aligned(w_in) && aligned(w_out) && aligned(y) &&
         aligned(pair_out);
}

// Grouping and both products; `sorted`, `tile_expert` and `tile_first` were made for tiles of 128
// rows. The grouped input lies in the rows of `pair_out` (half of each) until the second product
// writes them.
inline int moe_experts_tc(const void* hidden, int ld_hidden, const void* w_in, const void* w_out,
                          const int* sorted, const int* tile_expert, const int* tile_first,
                          int max_tiles, int rows, int experts, int top, int width, int ff,
                          MoeUnit unit, void* y, int ld_y, float* pair_out, int ld_out, int* status,
                          cudaStream_t stream) {
  const long long places = (long long)max_tiles * MT_ROWS;
  const long long most = 2LL * experts * (ff > width ? ff : width);
  if (places > 0x7fffffffLL || most > 0x7fffffffLL ||
      (long long)max_tiles * ((ff > width ? ff : width) / 128 + 1) > 0x7fffffffLL) {
    return AYK_TOO_LARGE;
  }
  CUtensorMap map_a, map_w, map_y, map_places, map_out;
  int r = make_map_128b(&map_a, pair_out, (uint64_t)rows * top, width, 2 * (uint64_t)ld_out,
                        MT_ROWS, 2);
  if (r != AYK_OK) return r;
  r = make_map_128b(&map_w, w_in, (uint64_t)experts * (unit.single ? 1 : 2) * ff, width, width,
                    MT_COLS / 2, 2);
  if (r != AYK_OK) return r;
  r = make_map_128b(&map_y, y, places, ff, ld_y, 32, 2);
  if (r != AYK_OK) return r;
  r = make_map_128b(&map_places, y, places, ff, ld_y, MT_ROWS, 2);
  if (r != AYK_OK) return r;
  r = make_map_128b(&map_out, w_out, (uint64_t)experts * width, ff, ff, MT_COLS / 2, 2);
  if (r != AYK_OK) return r;
  static const cudaError_t configured = [] {
    const cudaError_t e = cudaFuncSetAttribute(
        moe_tc_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, MT_DYNAMIC);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(moe_tc_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                MT_DYNAMIC);
  }();
  if (configured != cudaSuccess) return (int)configured;
  const auto grid = [&](int n, int tile_cols) {
    const long long tiles = (long long)max_tiles * ((n + tile_cols - 1) / tile_cols);
    return dim3((unsigned)(tiles < sm_count() ? tiles : sm_count()));
  };
  r = launch_kernel(moe_group_kernel, dim3(max_tiles, MT_ROWS / 8), dim3(256), 0, stream, 1,
                    (const __nv_bfloat16*)hidden, ld_hidden, sorted, tile_expert, tile_first, top,
                    width, (__nv_bfloat16*)pair_out, 2LL * ld_out);
  if (r != AYK_OK) return r;
  r = launch_kernel(moe_tc_kernel<0>, grid(ff, unit.single ? MT_COLS : MT_COLS / 2), dim3(192),
                    MT_DYNAMIC, stream, 1, map_a, map_w, map_y, sorted, tile_expert, tile_first, max_tiles,
                    width, ff, unit, (float*)nullptr, 0, status);
  if (r != AYK_OK) return r;
  return launch_kernel(moe_tc_kernel<1>, grid(width, MT_COLS), dim3(192), MT_DYNAMIC, stream, 1,
                       map_places, map_out, map_y, sorted, tile_expert, tile_first, max_tiles, ff,
                       width, unit, pair_out, ld_out, status);
}

}  // namespace ayk
