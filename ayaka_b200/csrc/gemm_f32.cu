// C[M,N] = A[M,K] * W[N,K]^T (+ bias, activation, residual) in float32 on the 5th-generation tensor
// cores, which have no 32-bit mode: every operand entry is taken apart into three bfloat16 numbers,
//   x = x1 + x2 + x3,   x1 = bf16(x),  x2 = bf16(x - x1),  x3 = bf16(x - x1 - x2),
// which between them hold its 24 bits and its range (to within 2^-27 |x|), and of the nine products of
// the parts the six that 32 bits can hold are added up:
//   a w = a1 w1 + (a1 w2 + a2 w1 + a1 w3 + a3 w1 + a2 w2)   to within 2^-26 |a w|.
// A product of two bfloat16 numbers is exact in fp32. The tensor core's own sums are kept short: 128 k are
// summed in tensor memory, products of different size apart, and those sums are added in fp32 registers,
// rounded to nearest. So the result is a true 32-bit product; against float64 its
// 2-norm is off by 1.0e-7 (K 768 to 1,024) and 1.1e-7 (3,072), that of FMAs in gemm_simt.cu by 1.8e-7 to
// 3.5e-7.
//
// The weights are the 128-row operand and a tile of NT rows of A the other one, so D[n, m] has a lane
// per output column whatever M is. Blocks of 32 k travel by TMA into a ring of raw fp32 tiles; all sixteen
// warps turn a block into bf16 tiles in the layout of TMA's 128-byte swizzle, two in turn: rows of W as
// w1 | w2 and w3 | nothing, the parts of A's rows below one another, so that three MMAs per 16 k form the
// six products, w1 [a1 a2 a3], w2 [a1 a2] and w3 a1, in accumulators of their own. One thread issues them;
// an MMA is short (N up to 240) and what a single thread does for each, descriptors above all, is what
// bounds a block, so both are kept few. Behind every fourth block the warps add the accumulators to their
// registers, lane n of 32 and a quarter of the rows each. One block barrier a block. K may be cut into stretches by N and K alone (f3_splits); their CTAs are a cluster and add up their sums in order
// through distributed shared memory. An element's sum has one order whatever M or the tile it falls in: a
// row's bits do not depend on its batch.
//
// An entry that is no number, infinite, or rounds to infinity makes x2 and so every sum it enters no
// number; entries below 2^-107 have parts that bfloat16 cannot hold, which may show in a sum that is
// itself tiny. Such an element (see f3_odd) is computed again with fp32 FMAs, so that what comes out is
// what 32-bit arithmetic gives.
//
// Every wait is bounded; a wait that runs out sets *status = AYK_WAIT_TIMEOUT, the CTA skips its stores,
// drains its copies, frees its tensor memory and returns.
#include "tensor_maps.cuh"

namespace ayk {

constexpr int F3_BM = 128, F3_BK = 32, F3_STAGES = 2;
constexpr int F3_SUM_K = 128;  // k of an accumulator
constexpr int F3_THREADS = 512;
constexpr int F3_SUM_BLOCKS = F3_SUM_K / F3_BK;
constexpr int F3_MAX_NT = 80;  // six accumulators in tensor memory

template <int NT>
struct F3Smem {
  static constexpr int ROWS = F3_BM + NT;
  // a stage, rows of 128 bytes: W's w1 | w2, W's w3 | nothing, A's a1 | nothing, a2 and a3
  static constexpr int A_OFFSET = 2 * F3_BM * 128;
  static constexpr int STAGE_BYTES = A_OFFSET + 3 * NT * 128;
  static constexpr int RAW_BYTES = ROWS * F3_BK * 4;
  static constexpr int RAW_OFFSET = F3_STAGES * STAGE_BYTES;
  static constexpr int LIMIT = 226 * 1024;
  static constexpr int FITS = (LIMIT - 1024 - 256 - RAW_OFFSET) / RAW_BYTES;
  static constexpr int RAW = FITS > 6 ? 6 : FITS;  // raw tiles in the ring
  static constexpr int BAR_OFFSET = RAW_OFFSET + RAW * RAW_BYTES;
  // raw_full[RAW], empty[STAGES], acc_full, then the tmem slot and the failure flag
  static constexpr int TOTAL = BAR_OFFSET + (RAW + F3_STAGES + 1) * 8 + 16;
  static constexpr int DYNAMIC = TOTAL + 1024;
  static_assert(RAW >= 3, "two blocks on their way while one is converted");
  static_assert(NT * F3_BM * 4 <= RAW_OFFSET, "the stages hold the partial sums at the end");
  static_assert(DYNAMIC <= 227 * 1024, "shared memory of an SM");
};

// Eight neighbouring entries as three rows of eight bfloat16 numbers.
__device__ __forceinline__ void f3_split(const float4& a, const float4& b, uint4 (&plane)[3]) {
  float x[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
  for (int p = 0; p < 3; ++p) {
    uint32_t u[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __nv_bfloat162 pair = __floats2bfloat162_rn(x[2 * i], x[2 * i + 1]);
      u[i] = *reinterpret_cast<const uint32_t*>(&pair);
      if (p < 2) {  // what is left (exact)
        x[2 * i] -= __uint_as_float(u[i] << 16);
        x[2 * i + 1] -= __uint_as_float(u[i] & 0xffff0000u);
      }
    }
    plane[p] = make_uint4(u[0], u[1], u[2], u[3]);
  }
}

// A sum that the parts may not give: no number, or so small that entries without all of their parts may
// have a share in it. (What an entry below 2^-107 lacks is at most 2^-134; beside factors above 2^40 it
// stays as it is.)
__device__ __forceinline__ bool f3_odd(float v) {
  return v != v || (fabsf(v) < 0x1p-60f && v != 0.f);
}
// One element with fp32 FMAs over k_first .. k_last.
__device__ __noinline__ float f3_plain(const float* a, const float* w, int k_first, int k_last) {
  float s = 0.f;
  for (int k = k_first; k < k_last; ++k) s = fmaf(a[k], w[k], s);
  return s;
}

__device__ __forceinline__ void f3_ld_32x4(uint32_t taddr, uint32_t* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
               : "r"(taddr)
               : "memory");
}

// grid (weight tiles * splits, row tiles), clusters of `splits` along x.
template <int NT>
__global__ void __launch_bounds__(F3_THREADS, 1)
gemm_f32_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a,
                const float* __restrict__ a, int lda, const float* __restrict__ w, int ldw,
                const float* __restrict__ bias, float* __restrict__ out, int ldo, int M, int N,
                int K, int act, int residual, int splits, int k_split,
                int* __restrict__ status) {
  using L = F3Smem<NT>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
  uint64_t* raw_full = reinterpret_cast<uint64_t*>(smem + L::BAR_OFFSET);
  uint64_t* empty = raw_full + L::RAW;
  uint64_t* acc_full = empty + F3_STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
  volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);
  // the accumulators of w1, w2 and w3
  constexpr int D2 = (3 * NT + 31) / 32 * 32, D3 = D2 + 2 * NT, D_END = D3 + (NT + 31) / 32 * 32;
  constexpr uint32_t TMEM_COLS = D_END <= 128 ? 128 : (D_END <= 256 ? 256 : 512);
  static_assert(D_END <= 512 && D2 % 32 == 0 && D3 % 32 == 0, "tensor memory");
  constexpr int NQ = NT / 4;  // rows of a warp's sums

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = splits > 1 ? (int)(blockIdx.x % splits) : 0;
  const int n0 = (int)(blockIdx.x / splits) * F3_BM, m0 = blockIdx.y * NT;
  const int k_first = rank * k_split, k_last = min(K, k_first + k_split);
  const int num_kb = (k_last - k_first + F3_BK - 1) / F3_BK;  // blocks

  if (tid == 0) {
    for (int s = 0; s < L::RAW; ++s) mbar_init(&raw_full[s], 1);
    for (int s = 0; s < F3_STAGES; ++s) mbar_init(&empty[s], 1);
    mbar_init(acc_full, 1);
    *failed = 0;
    mbar_fence_init();
    tma_prefetch_map(&map_w);
    tma_prefetch_map(&map_a);
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

  int issued = 0;  // (thread 32) blocks whose copies it has started
  auto raw_tile = [&](int slot) { return smem + L::RAW_OFFSET + slot * L::RAW_BYTES; };
  auto bring_w = [&](int kb, int slot) {
    mbar_expect_tx(&raw_full[slot], L::RAW_BYTES);
    tma_load_2d(raw_tile(slot), &map_w, &raw_full[slot], k_first + kb * F3_BK, n0);
  };
  auto bring_a = [&](int kb, int slot) {
    tma_load_2d(raw_tile(slot) + F3_BM * F3_BK * 4, &map_a, &raw_full[slot], k_first + kb * F3_BK, m0);
    issued = kb + 1;
  };
  if (tid == 32) {
    const int ahead = num_kb < L::RAW ? num_kb : L::RAW;
    for (int kb = 0; kb < ahead; ++kb) bring_w(kb, kb);  // weights: ahead of the dependency wait
    pdl_wait();
    for (int kb = 0; kb < ahead; ++kb) bring_a(kb, kb);
  }
  __syncwarp();

  const int quarter = warp & 3, part = warp >> 2;
  const int n = n0 + quarter * 32 + lane;  // this lane's output column
  float acc[NQ];
#pragma unroll
  for (int j = 0; j < NQ; ++j) acc[j] = 0.f;
  uint32_t sums = 0;  // accumulators added so far
  auto add = [&]() {  // the accumulators to the sums: lane n, rows part * NQ ..
    if (*failed == 0 && !mbar_wait(acc_full, sums & 1)) *failed = 1;
    ++sums;
    __syncwarp();
    tc_fence_after();
    const uint32_t from = tmem_base + (uint32_t)(part * NQ) + ((uint32_t)(quarter * 32) << 16);
#pragma unroll
    for (int j = 0; j < NQ; j += 4) {
      uint32_t x[6][4];
      f3_ld_32x4(from + j, x[0]);
      f3_ld_32x4(from + NT + j, x[1]);
      f3_ld_32x4(from + D2 + j, x[2]);
      f3_ld_32x4(from + 2 * NT + j, x[3]);
      f3_ld_32x4(from + D2 + NT + j, x[4]);
      f3_ld_32x4(from + D3 + j, x[5]);
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float least = __uint_as_float(x[3][e]) + __uint_as_float(x[4][e]) + __uint_as_float(x[5][e]);
        const float rest = __uint_as_float(x[1][e]) + __uint_as_float(x[2][e]) + least;
        acc[j + e] += __uint_as_float(x[0][e]) + rest;
      }
    }
    tc_fence_before();
  };
  // descriptors: the low words differ by where a tile starts (in 16 bytes), the high ones not
  const uint64_t desc0 = umma_desc_k128(smem, 0);
  auto desc = [&](uint32_t bytes) {
    return (desc0 & 0xffffffff00000000ull) | ((uint32_t)desc0 + (bytes >> 4));
  };
  constexpr uint32_t idesc1 = umma_idesc_bf16(F3_BM, 3 * NT), idesc2 = umma_idesc_bf16(F3_BM, 2 * NT),
                     idesc3 = umma_idesc_bf16(F3_BM, NT);
  // a thread: 8 neighbouring k (piece p of 4) of row r of W and, for the first NT, of A
  const int r = tid >> 2, p = tid & 3, x = r & 7;
  const bool odd_row = x & 1;
  const uint32_t raw0 = (uint32_t)(((2 * p) ^ x) << 4), raw1 = (uint32_t)(((2 * p + 1) ^ x) << 4);
  // (of W, odd rows store x2 first: two rows side by side in different halves of the banks)
  const uint32_t to0 = (uint32_t)((((odd_row ? 4 : 0) + p) ^ x) << 4);
  const uint32_t to1 = (uint32_t)((((odd_row ? 0 : 4) + p) ^ x) << 4);
  const uint32_t to2 = (uint32_t)((p ^ x) << 4);
  int slot = 0;          // of the raw ring
  uint32_t round = 0;    // parity of the ring's turn
  for (int kb = 0; kb < num_kb; ++kb) {
    const int s = kb & 1;
    if (*failed == 0 && (!mbar_wait(&raw_full[slot], round) ||
                         (kb >= F3_STAGES && !mbar_wait(&empty[s], ((kb >> 1) & 1) ^ 1)))) {
      *failed = 1;
    }
    const uint8_t* raw = raw_tile(slot) + r * 128;
    uint8_t* tile = smem + s * L::STAGE_BYTES + r * 128;
    uint4 plane[3];
    f3_split(*reinterpret_cast<const float4*>(raw + raw0), *reinterpret_cast<const float4*>(raw + raw1),
             plane);
    *reinterpret_cast<uint4*>(tile + to0) = odd_row ? plane[1] : plane[0];
    *reinterpret_cast<uint4*>(tile + to1) = odd_row ? plane[0] : plane[1];
    *reinterpret_cast<uint4*>(tile + F3_BM * 128 + to2) = plane[2];
    if (r < NT) {
      f3_split(*reinterpret_cast<const float4*>(raw + F3_BM * 128 + raw0),
               *reinterpret_cast<const float4*>(raw + F3_BM * 128 + raw1), plane);
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        *reinterpret_cast<uint4*>(tile + L::A_OFFSET + q * NT * 128 + to2) = plane[q];
      }
    }
    fence_proxy_async_shared();
    // (before the accumulators begin anew; their last MMAs ran under this block's conversion)
    const bool begins = kb % F3_SUM_BLOCKS == 0;
    if (begins && kb > 0) add();
    __syncthreads();  // the block is converted
    if (tid == 0) {
      tc_fence_after();
      const uint32_t w12 = s * L::STAGE_BYTES, w3 = w12 + F3_BM * 128, a1 = w12 + L::A_OFFSET;
#pragma unroll
      for (int k = 0; k < F3_BK / 16; ++k) {
        const uint32_t more = !begins || k != 0;
        umma_f16(tmem_base, desc(w12 + k * 32), desc(a1 + k * 32), idesc1, more);
        umma_f16(tmem_base + D2, desc(w12 + 64 + k * 32), desc(a1 + k * 32), idesc2, more);
        umma_f16(tmem_base + D3, desc(w3 + k * 32), desc(a1 + k * 32), idesc3, more);
      }
      umma_commit(&empty[s]);
      if (kb % F3_SUM_BLOCKS == F3_SUM_BLOCKS - 1 || kb + 1 == num_kb) umma_commit(acc_full);
    }
    if (tid == 32 && kb + L::RAW < num_kb && *failed == 0) {  // (every warp has read the raw tile)
      bring_w(kb + L::RAW, slot);
      bring_a(kb + L::RAW, slot);
    }
    __syncwarp();
    if (++slot == L::RAW) {
      slot = 0;
      round ^= 1;
    }
  }
  add();
  pdl_wait_for(a, out);

  // ---- this stretch's sums; what is odd once more
  {
    bool odd = false;
#pragma unroll
    for (int j = 0; j < NQ; ++j) odd |= f3_odd(acc[j]);
    if (odd && n < N && *failed == 0) {
      float again[NQ];
#pragma unroll
      for (int j = 0; j < NQ; ++j) again[j] = acc[j];
#pragma unroll 1
      for (int j = 0; j < NQ; ++j) {
        const int m = m0 + part * NQ + j;
        if (m < M && f3_odd(again[j])) {
          again[j] = f3_plain(a + (size_t)m * lda, w + (size_t)n * ldw, k_first, k_last);
        }
      }
#pragma unroll
      for (int j = 0; j < NQ; ++j) acc[j] = again[j];
    }
    __syncwarp();
  }
  // Into shared memory (every MMA has read its operands, the last accumulator was complete: the stages are
  // free), and from there, added up over the stretches, a row of 128 columns a time. (One small loop: with
  // the activation unrolled over a lane's own sums the kernel waited for its code.)
  float* partial = reinterpret_cast<float*>(smem);  // [NT][128]
#pragma unroll
  for (int j = 0; j < NQ; ++j) partial[(part * NQ + j) * F3_BM + quarter * 32 + lane] = acc[j];
  if (splits > 1) {
    cluster_sync_all();
  } else {
    __syncthreads();
  }
  const int column = n0 + (tid & 127);
  if (*failed == 0 && column < N) {
    const float b = bias != nullptr ? __ldg(bias + column) : 0.f;
    const int step = splits * (F3_THREADS / 128), rows = min(NT, M - m0);
#pragma unroll 1
    for (int row = rank + splits * (tid >> 7); row < rows; row += 4 * step) {
      float v[4], old[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int at = min(row + i * step, NT - 1);
        v[i] = partial[at * F3_BM + (tid & 127)];
        old[i] = residual && row + i * step < rows
                     ? out[(size_t)(m0 + at) * ldo + column] : 0.f;
      }
      if (splits > 1) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float* mine = partial + min(row + i * step, NT - 1) * F3_BM + (tid & 127);
          v[i] = ld_peer_f32(mine, 0);
          for (int r = 1; r < splits; ++r) v[i] += ld_peer_f32(mine, r);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] += b;
      if (!residual) activate_all<false>(v, act);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (row + i * step < rows) out[(size_t)(m0 + row + i * step) * ldo + column] = old[i] + v[i];
      }
    }
  }
  __syncwarp();
  if (splits > 1) cluster_sync_all();  // nobody leaves while a peer may still read its sums

  tc_fence_before();
  __syncthreads();
  if (*failed != 0 && tid == 32) {
    // copies this thread started may still be landing: wait for each, bounded
    for (int kb = issued > L::RAW ? issued - L::RAW : 0; kb < issued; ++kb) {
      mbar_wait(&raw_full[kb % L::RAW], (kb / L::RAW) & 1);
    }
    atomicExch(status, AYK_WAIT_TIMEOUT);
  }
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem_base, TMEM_COLS);
}

// Stretches of K, by N and K alone: about 20 CTAs a tile of rows (what seven tiles of rows can fill the
// device with) as long as a stretch has at least 256 k.
inline int f3_splits(int N, int K) {
  const int tiles = (N + F3_BM - 1) / F3_BM, blocks = (K + F3_SUM_K - 1) / F3_SUM_K;
  int splits = 1;
  while (splits < 8 && tiles * (splits + 1) <= 20 && blocks >= 2 * (splits + 1)) ++splits;
  const int each = (blocks + splits - 1) / splits;
  return (blocks + each - 1) / each;  // (no stretch without a block)
}

// Rows of a tile: the width with the least (rounds over the SMs) x (time of a CTA).
inline int f3_rows(int M, int ctas, int blocks) {
  const int sms = sm_count();
  long long best = -1;
  int best_nt = F3_MAX_NT;
  for (int tiles = (M + F3_MAX_NT - 1) / F3_MAX_NT, tried = 0; tried < 8; ++tiles, ++tried) {
    const int nt = ((M + tiles - 1) / tiles + 15) / 16 * 16;
    const long long rounds = ((long long)ctas * ((M + nt - 1) / nt) + sms - 1) / sms;
    const long long cost = rounds * (5000 + (long long)blocks * (1000 + 10 * nt));
    if (best < 0 || cost < best) {
      best = cost;
      best_nt = nt;
    }
    if (nt == 16) break;
  }
  return best_nt;
}

template <int NT>
int launch_gemm_f32(const float* a, int lda, const float* w, int ldw, const float* bias, float* out,
                    int ldo, int M, int N, int K, int act, int residual, int splits, int k_split,
                    int* status, cudaStream_t stream) {
  using L = F3Smem<NT>;
  CUtensorMap map_w, map_a;
  int r = cached_map(w, (uint64_t)N, (uint64_t)K, (uint64_t)ldw, F3_BM, &map_w, 4);
  if (r != AYK_OK) return r;
  r = cached_map(a, (uint64_t)M, (uint64_t)K, (uint64_t)lda, NT, &map_a, 4);
  if (r != AYK_OK) return r;
  static const cudaError_t allowed = cudaFuncSetAttribute(
      gemm_f32_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::DYNAMIC);
  if (allowed != cudaSuccess) return (int)allowed;
  const dim3 grid((N + F3_BM - 1) / F3_BM * splits, (M + NT - 1) / NT);
  return launch_kernel_x(gemm_f32_kernel<NT>, grid, dim3(F3_THREADS), L::DYNAMIC, stream, splits,
                         map_w, map_a, a, lda, w, ldw, bias, out, ldo, M, N, K, act, residual, splits,
                         k_split, status);
}

}  // namespace ayk

AYK_API void ayk_set_pdl(int on) { ayk::pdl_enabled() = on; }

// `residual` != 0: out is added to. `tile_rows`: 0 chooses, else 16, 32, ... 80 rows of A a tile (for
// tests). AYK_NOT_TAKEN, and nothing ran: operands whose rows do not start on 16 bytes, or more row tiles
// than a grid counts; the FMA kernel of gemm_simt.cu takes any.
AYK_API int ayk_gemm_f32(const float* a, int lda, const float* w, int ldw, const float* bias,
                         float* out, int ldo, int M, int N, int K, int act, int residual,
                         int tile_rows, int* status, void* stream) {
  using namespace ayk;
  if (M == 0 || N == 0) return AYK_OK;
  if (M < 0 || N < 0 || K < 1 || lda < K || ldw < K || ldo < N || status == nullptr ||
      act < ACT_NONE || act > ACT_RELU_SQUARED || (residual && act != ACT_NONE) || tile_rows < 0 ||
      tile_rows > F3_MAX_NT || tile_rows % 16) {
    return AYK_BAD_ARGUMENT;
  }
  if (lda % 4 || ldw % 4 || (uintptr_t)a % 16 || (uintptr_t)w % 16) return AYK_NOT_TAKEN;
  const int blocks = (K + F3_SUM_K - 1) / F3_SUM_K, splits = f3_splits(N, K);
  const int each = (blocks + splits - 1) / splits;
  const long long ctas = (long long)((N + F3_BM - 1) / F3_BM) * splits;
  if (ctas > 0x7fffffffLL) return AYK_NOT_TAKEN;
  const int nt = tile_rows ? tile_rows : f3_rows(M, (int)ctas, each);
  if ((M + nt - 1) / nt > 65535) return AYK_NOT_TAKEN;
#define AYK_F3(NT)                                                                               \
  case NT:                                                                                       \
    return launch_gemm_f32<NT>(a, lda, w, ldw, bias, out, ldo, M, N, K, act, residual, splits,   \
                               each * F3_SUM_K, status, (cudaStream_t)stream)
  switch (nt) {
    AYK_F3(16);
    AYK_F3(32);
    AYK_F3(48);
    AYK_F3(64);
    AYK_F3(80);
  }
#undef AYK_F3
  return AYK_BAD_ARGUMENT;
}
