// Causal attention for prompt portions in bfloat16 over the paged cache with both products on the
// 5th-generation tensor cores, for what attention_prefill_tc.cu does not serve: head sizes 64 and
// 128 with a window's kept first keys, a gate or a sink, and latent rows of 256 entries that are
// keys and values at once (SAME). Options as in attention_prefill.cu: `window`, `keep_first`, `gate`
// (the result times the sigmoid of one raw gate per entry), `sink` (one more entry of the softmax's
// denominator per head).
//
// A CTA owns 128 consecutive query rows of one request and one head and walks that request's keys 64
// at a time: first the blocks of kept keys, then from the window's first block up to the tile's last
// row. Six warps:
//   warps 0-3  softmax: a thread owns a row, whose 64 scores of a block it reads from tensor memory
//              into registers at once. The running reference moves only when a block's maximum
//              exceeds it by more than 8 (log2 units), so that most blocks do not touch the
//              accumulator; P is written to shared memory as bf16 in the layout the tensor core
//              reads;
//   warp 4     one thread issues S = Q K^T (two score tiles, so that the next block's scores are
//              there when a softmax ends) and O += P V (V as stored, [key][64 entries], MN-major);
//   warp 5     fetches Q (one TMA box per 64 entries of the head), then the K and V blocks by TMA, a
//              box per page and 64 entries, into a ring in the order in which they are used: K0, K1,
//              V0, K2, V1, ... (SAME: one block serves both products).
// Bound by the softmax of 64 keys a turn, which is why two CTAs share an SM where they fit (head sizes
// 64 and 128: 97 KB and 256 tensor-memory columns each): the tensor pipe is active for 27 % of the time
// at head size 128 and 21 % over latent rows, issue slots are used for 37 % and 19 %.
// Rows of a value block that no row of the tile may see are zeroed after they land (their pages may be
// gone, and 0 * NaN would poison the sum); keys out of sight are masked in the scores. Blocks are
// aligned to absolute positions, so a row's result does not depend on how the prompt was cut.
// Every wait is bounded (tc_common.cuh); one that runs out sets the status word.
//
// Measured on a B200 against the warp-level kernel: 16 heads. Head size 128: 4,096 rows
// 457 -> 133 microseconds; four requests of 4,096 rows together, window 512, 64 kept keys and a gate
// 188 -> 78; the same over latent rows without kept keys 201 -> 82; head size 64 as the first 88 -> 57.
#include "tc_common.cuh"

namespace ayk {

constexpr int FW_BM = 128, FW_BN = 64, FW_THREADS = 192;
constexpr int FW_Q_TILE = FW_BM * 128, FW_KV_TILE = FW_BN * 128;  // bytes per 64 entries of the head
constexpr float FW_LAZY = 8.f;

template <int D, bool SAME>
struct FwShape {
  static constexpr int TILES = D / 64;
  static constexpr int ENTRIES = 3;  // blocks in the ring
  static constexpr int ENTRY = TILES * FW_KV_TILE;
  static constexpr int Q = 0;
  static constexpr int RING = Q + TILES * FW_Q_TILE;
  static constexpr int P = RING + ENTRIES * ENTRY;
  static constexpr int BAR = P + FW_Q_TILE;
  // q_full, p_full, pv_done, land; s_full[2]; full[ENTRIES], empty[ENTRIES]
  static constexpr int BARS = 6 + 2 * ENTRIES;
  static constexpr int DYNAMIC = BAR + BARS * 8 + 16 + 1024;
  static constexpr uint32_t O_COL = 2 * FW_BN;
  static constexpr uint32_t TMEM_COLS = O_COL + D <= 256 ? 256 : 512;
};

__device__ __forceinline__ void fw_tmem_st_32x32(uint32_t taddr, const uint32_t* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(
          taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
      "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]),
      "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]),
      "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]),
      "r"(v[29]), "r"(v[30]), "r"(v[31])
      : "memory");
}
__device__ __forceinline__ void fw_tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ float fw_exp2(float x) {  // 2 ulp; exp2(-inf) = 0
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 16 rows (keys) of an MN-major operand: rows of 128 bytes with the 128-byte swizzle.
__device__ __forceinline__ uint64_t fw_desc_mn128(const void* tile) {
  const uint32_t addr = smem_u32(tile);
  uint64_t desc = 0;
  desc |= (uint64_t)((addr & 0x3FFFFu) >> 4);
  desc |= (uint64_t)1 << 16;
  desc |= (uint64_t)(1024 >> 4) << 32;
  desc |= (uint64_t)1 << 46;
  desc |= (uint64_t)2 << 61;
  return desc;
}
__device__ __forceinline__ uint32_t fw_pack(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}

template <int D, bool SAME>
__global__ void __launch_bounds__(FW_THREADS)
attention_prefill_wide_kernel(const __grid_constant__ CUtensorMap map_q,
                              const __grid_constant__ CUtensorMap map_k,
                              const __grid_constant__ CUtensorMap map_v, int box_rows,
                              const int* __restrict__ block_table, int table_stride,
                              const int* __restrict__ row_start, const int* __restrict__ kv_len,
                              __nv_bfloat16* __restrict__ out, int ld_out, int num_requests,
                              int num_kv_heads, int group, int page_size, int page_shift,
                              float scale, int window, int keep_first, int total_tiles,
                              const float* __restrict__ gate, int ld_gate,
                              const float* __restrict__ sink, int* __restrict__ status) {
  using L = FwShape<D, SAME>;
  constexpr int T = L::TILES, E = L::ENTRIES;
  extern __shared__ uint8_t fw_raw[];
  uint8_t* smem = fw_raw + ((1024 - (smem_u32(fw_raw) & 1023)) & 1023);
  uint64_t* q_full = reinterpret_cast<uint64_t*>(smem + L::BAR);
  uint64_t* p_full = q_full + 1;   // 4 arrivals: S has been read, P is in shared memory
  uint64_t* pv_done = p_full + 1;  // MMA commit: O += P V has finished
  uint64_t* land = pv_done + 1;    // a block whose rows need zeroing lands here first
  uint64_t* s_full = land + 1;     // [2] MMA commit: S is in tensor memory
  uint64_t* full = s_full + 2;     // [ring]
  uint64_t* empty = full + E;      // [ring] MMA commit: the block has been read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(empty + E);
  volatile int* failed = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    mbar_init(p_full, 4);
    mbar_init(pv_done, 1);
    mbar_init(land, 1);
    mbar_init(&s_full[0], 1);
    mbar_init(&s_full[1], 1);
    for (int s = 0; s < E; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    *failed = 0;
    mbar_fence_init();
  }
  if (warp == 4) {
    tmem_alloc(tmem_slot, L::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();
  pdl_wait_for(gate, out);

  // Which request and which tile of it: heads along grid.x, tiles along grid.y from the last one
  // down (the longest first).
  int tile = total_tiles - 1 - (int)blockIdx.y, req = 0, rows_b = 0;
  for (; req < num_requests; ++req) {
    rows_b = row_start[req + 1] - row_start[req];
    const int tiles = (rows_b + FW_BM - 1) / FW_BM;
    if (tile < tiles) break;
    tile -= tiles;
  }
  const int head = blockIdx.x, kv_head = head / group;
  bool work = req < num_requests;
  int first_row = 0, nrows = 0, length = 0;
  if (work) {
    first_row = row_start[req] + tile * FW_BM;
    nrows = rows_b - tile * FW_BM < FW_BM ? rows_b - tile * FW_BM : FW_BM;
    length = kv_len[req];
    if (length == 0) {  // a padding request: zeros
      for (int i = threadIdx.x; i < nrows * (D / 8); i += FW_THREADS) {
        *reinterpret_cast<uint4*>(out + (size_t)(first_row + i / (D / 8)) * ld_out + head * D +
                                  (i % (D / 8)) * 8) = make_uint4(0u, 0u, 0u, 0u);
      }
      work = false;
    }
  }
  if (work) {
    const int pos0 = length - rows_b + tile * FW_BM;  // position of the tile's first row
    const int last_key = pos0 + nrows - 1;
    const int lo_min = (window > 0 && pos0 - window + 1 > 0) ? pos0 - window + 1 : 0;
    const int block_lo = lo_min / FW_BN;
    // kept first keys that the window of the tile's first row has left behind: their blocks come
    // first (those that the window's walk does not reach anyway)
    const int keep = window > 0 ? keep_first : 0;
    const int kept = keep < lo_min ? keep : lo_min;
    int kept_blocks = (kept + FW_BN - 1) / FW_BN;
    if (kept_blocks > block_lo) kept_blocks = block_lo;
    const int turns = kept_blocks + last_key / FW_BN - block_lo + 1;
    auto first_key = [&](int turn) {
      return (turn < kept_blocks ? turn : block_lo + turn - kept_blocks) * FW_BN;
    };
    // the ring's place in the order of use of a turn's keys and values
    auto k_place = [&](int i) { return SAME ? i : (i == 0 ? 0 : 2 * i - 1); };
    auto v_place = [&](int i) { return SAME ? i : (i + 1 < turns ? 2 * i + 2 : 2 * i + 1); };

    if (warp == 5) {
      // ---- producer
      const int* table = block_table + (size_t)req * table_stride;
      if (lane == 0) {
        mbar_expect_tx(q_full, T * FW_Q_TILE);
        for (int t = 0; t < T; ++t) {
          tma_load_2d(smem + L::Q + t * FW_Q_TILE, &map_q, q_full, head * D + t * 64, first_row);
        }
      }
      const int boxes = FW_BN / box_rows, places = SAME ? turns : 2 * turns;
      const uint32_t box_bytes = (uint32_t)box_rows * 128u;
      bool ok = true;
      int issued = 0, landed = 0;
      for (int n = 0; n < places && ok; ++n) {
        // place n: K of turn (n + 1) / 2 for odd n (and 0), V of turn n / 2 - 1 for even n; the
        // last place is V of the last turn
        const bool values = !SAME && n > 0 && ((n & 1) == 0 || n == places - 1);
        const int turn = SAME ? n : (values ? (n == places - 1 ? turns - 1 : n / 2 - 1)
                                            : (n + 1) / 2);
        const int s = n % E;
        if (n >= E) {
          if (lane == 0) ok = mbar_wait(&empty[s], (uint32_t)(n / E - 1) & 1u);
          ok = __shfl_sync(0xffffffffu, ok, 0);
          if (!ok) break;
        }
        const int key0 = first_key(turn), key = key0 + lane * box_rows;
        const bool fetch = lane < boxes && key <= last_key &&
                           (key + box_rows - 1 >= lo_min || key < keep);
        const uint32_t count = (uint32_t)__popc(__ballot_sync(0xffffffffu, fetch));
        // (a block of kept keys may hold others too)
        const bool fix = (SAME || values) &&
                         (key0 + FW_BN - 1 > last_key || (key0 < lo_min && key0 + FW_BN > keep));
        uint64_t* lands = fix ? land : &full[s];
        uint8_t* entry = smem + L::RING + s * L::ENTRY;
        if (lane == 0) mbar_expect_tx(lands, count * box_bytes * T);
        __syncwarp();
        if (fetch) {
          const int index = page_shift >= 0 ? key >> page_shift : key / page_size;
          const int slot = page_shift >= 0 ? key & (page_size - 1) : key % page_size;
          const int row = (table[index] * num_kv_heads + kv_head) * page_size + slot;
          for (int t = 0; t < T; ++t) {
            tma_load_2d(entry + t * FW_KV_TILE + lane * box_bytes, values ? &map_v : &map_k, lands,
                        t * 64, row);
          }
        }
        issued = n + 1;
        if (fix) {
          if (lane == 0) ok = mbar_wait(land, (uint32_t)landed & 1u);
          ok = __shfl_sync(0xffffffffu, ok, 0);
          if (!ok) break;
          ++landed;
          for (int i = lane; i < FW_BN * 8; i += 32) {
            const int k = key0 + (i >> 3);
            if (k > last_key || (k < lo_min && k >= keep)) {
              for (int t = 0; t < T; ++t) {
                *reinterpret_cast<uint4*>(entry + t * FW_KV_TILE + (i >> 3) * 128 +
                                          ((i & 7) << 4)) = make_uint4(0u, 0u, 0u, 0u);
              }
            }
          }
          fence_proxy_async_shared();
          __syncwarp();
          if (lane == 0) mbar_arrive(&full[s]);
        }
      }
      if (lane == 0) {  // nothing of this warp's is in flight when it leaves
        if (!ok) *failed = 1;
        mbar_wait(q_full, 0);
        for (int n = issued > E ? issued - E : 0; n < issued && ok; ++n) {
          mbar_wait(&full[n % E], (uint32_t)(n / E) & 1u);
        }
      }
      __syncwarp();
    } else if (warp == 4) {
      // ---- MMA issuer
      if (lane == 0) {
        constexpr uint32_t idesc_s = umma_idesc_bf16(FW_BM, FW_BN);
        constexpr uint32_t idesc_o = umma_idesc_bf16(FW_BM, 64) | (1u << 16);  // B: MN-major
        const uint8_t* q_s = smem + L::Q;
        const uint8_t* p_s = smem + L::P;
        const int places = SAME ? turns : 2 * turns;
        // Only a place that the producer fills again is handed back: nobody waits for the last ones,
        // and an arrival of theirs could come when the CTA has left and the next one owns the memory.
        auto hand_back = [&](int n) {
          if (n + E < places) umma_commit(&empty[n % E]);
        };
        bool ok = mbar_wait(q_full, 0);
        auto scores = [&](int i) {
          const int n = k_place(i), s = n % E;
          if (!mbar_wait(&full[s], (uint32_t)(n / E) & 1u)) return false;
          tc_fence_after();
          const uint8_t* k_tile = smem + L::RING + s * L::ENTRY;
#pragma unroll
          for (int t = 0; t < T; ++t) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              umma_f16(tmem_base + (uint32_t)((i & 1) * FW_BN),
                       umma_desc_k128(q_s + t * FW_Q_TILE, k * 32),
                       umma_desc_k128(k_tile + t * FW_KV_TILE, k * 32), idesc_s, (t | k) != 0);
            }
          }
          umma_commit(&s_full[i & 1]);
          if (!SAME) hand_back(n);
          return true;
        };
        if (ok) ok = scores(0);
        for (int i = 0; i < turns && ok; ++i) {
          // (the score tile of turn i + 1 was read before P of turn i - 1 was handed over)
          if (i + 1 < turns) ok = scores(i + 1);
          if (ok) ok = mbar_wait(p_full, (uint32_t)i & 1u);
          const int n = v_place(i), s = n % E;
          if (ok) ok = mbar_wait(&full[s], (uint32_t)(n / E) & 1u);
          if (!ok) break;
          tc_fence_after();
          const uint8_t* v_tile = smem + L::RING + s * L::ENTRY;
#pragma unroll
          for (int k = 0; k < FW_BN / 16; ++k) {
#pragma unroll
            for (int t = 0; t < T; ++t) {
              umma_f16(tmem_base + L::O_COL + (uint32_t)(t * 64), umma_desc_k128(p_s, k * 32),
                       fw_desc_mn128(v_tile + t * FW_KV_TILE + k * 16 * 128), idesc_o,
                       (i | k) != 0);
            }
          }
          umma_commit(pv_done);
          hand_back(n);
        }
        if (!ok) *failed = 1;
      }
      __syncwarp();
    } else {
      // ---- softmax
      const int r = threadIdx.x;
      const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
      const uint32_t o_acc = tmem_base + L::O_COL + lane_base;
      const int pos = pos0 + r;
      const int after = window > 0 ? pos - window : -2147483647 - 1;  // keys > after are seen
      const float scale2 = scale * 1.4426950408889634f;  // scores in units of log2
      float ref = -INFINITY, sum = 0.f;
      const int swz = r & 7;
      uint8_t* p_row = smem + L::P + r * 128;
      bool ok = true;
      auto wait_one = [&](uint64_t* bar, uint32_t parity) {
        if (lane == 0) ok = mbar_wait(bar, parity);
        ok = __shfl_sync(0xffffffffu, ok, 0);
        tc_fence_after();
      };
      for (int i = 0; i < turns; ++i) {
        const int key0 = first_key(i);
        wait_one(&s_full[i & 1], (uint32_t)(i >> 1) & 1u);
        if (!ok) break;
        uint32_t raw[64];
        tmem_ld_32x32(tmem_base + (uint32_t)((i & 1) * FW_BN) + lane_base, raw);
        tmem_ld_32x32(tmem_base + (uint32_t)((i & 1) * FW_BN + 32) + lane_base, raw + 32);
        tmem_ld_wait();
        // a block that every row of the tile sees whole has nothing to mask
        const bool all_seen = key0 + FW_BN - 1 <= pos0 &&
                              (window == 0 || key0 > pos0 + FW_BM - 1 - window);
        float top0 = -INFINITY, top1 = -INFINITY;
        if (all_seen) {
#pragma unroll
          for (int c = 0; c < 64; c += 2) {
            top0 = fmaxf(top0, __uint_as_float(raw[c]));
            top1 = fmaxf(top1, __uint_as_float(raw[c + 1]));
          }
        } else {
#pragma unroll
          for (int c = 0; c < 64; ++c) {
            const int key = key0 + c;
            const bool seen = (key <= pos) & ((key > after) | (key < keep));
            raw[c] = seen ? raw[c] : 0xff800000u;  // -inf
          }
#pragma unroll
          for (int c = 0; c < 64; c += 2) {
            top0 = fmaxf(top0, __uint_as_float(raw[c]));
            top1 = fmaxf(top1, __uint_as_float(raw[c + 1]));
          }
        }
        const float top = fmaxf(top0, top1) * scale2;
        const bool moves = ref != -INFINITY && top > ref + FW_LAZY;
        float alpha = 1.f;
        if (moves) alpha = fw_exp2(ref - top);
        if (moves || ref == -INFINITY) ref = top;  // (-inf while the row has seen no key)
        if (i > 0) {  // P's space is free, and the accumulator whole
          wait_one(pv_done, (uint32_t)(i - 1) & 1u);
          if (!ok) break;
          if (__any_sync(0xffffffffu, moves)) {
#pragma unroll 1
            for (int c = 0; c < D / 32; ++c) {
              uint32_t v[32];
              tmem_ld_32x32(o_acc + (uint32_t)(c * 32), v);
              tmem_ld_wait();
#pragma unroll
              for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) * alpha);
              fw_tmem_st_32x32(o_acc + (uint32_t)(c * 32), v);
            }
            fw_tmem_st_wait();
            sum *= alpha;
          }
        }
        const float offset = ref == -INFINITY ? 0.f : -ref;
        float part0 = 0.f, part1 = 0.f;
#pragma unroll
        for (int h = 0; h < 8; ++h) {  // eight keys a 16-byte piece
          float p[8];
#pragma unroll
          for (int e = 0; e < 8; e += 2) {
            p[e] = fw_exp2(fmaf(__uint_as_float(raw[h * 8 + e]), scale2, offset));
            p[e + 1] = fw_exp2(fmaf(__uint_as_float(raw[h * 8 + e + 1]), scale2, offset));
            part0 += p[e];
            part1 += p[e + 1];
          }
          *reinterpret_cast<uint4*>(p_row + ((h ^ swz) << 4)) =
              make_uint4(fw_pack(p[0], p[1]), fw_pack(p[2], p[3]), fw_pack(p[4], p[5]),
                         fw_pack(p[6], p[7]));
        }
        sum += part0 + part1;
        tc_fence_before();
        fence_proxy_async_shared();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full);
      }
      if (ok) wait_one(pv_done, (uint32_t)(turns - 1) & 1u);
      if (ok) {
        float inv = 1.f / sum;
        if (sink != nullptr) {
          const float sink2 = sink[head] * 1.4426950408889634f, most = fmaxf(ref, sink2);
          const float corr = exp2f(ref - most);
          inv = corr / (sum * corr + exp2f(sink2 - most));
        }
        __nv_bfloat16* dst = out + (size_t)(first_row + r) * ld_out + head * D;
        const float* g = gate != nullptr ? gate + (size_t)(first_row + r) * ld_gate + head * D
                                         : nullptr;
#pragma unroll 1
        for (int c = 0; c < D / 32; ++c) {
          uint32_t v[32];
          tmem_ld_32x32(o_acc + (uint32_t)(c * 32), v);
          tmem_ld_wait();
          if (r < nrows) {
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              float x[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) x[e] = __uint_as_float(v[h * 8 + e]) * inv;
              if (g != nullptr) {
                const float4 a = *reinterpret_cast<const float4*>(g + c * 32 + h * 8);
                const float4 b = *reinterpret_cast<const float4*>(g + c * 32 + h * 8 + 4);
                const float z[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
                for (int e = 0; e < 8; ++e) x[e] /= 1.f + expf(-z[e]);
              }
              *reinterpret_cast<uint4*>(dst + c * 32 + h * 8) =
                  make_uint4(fw_pack(x[0], x[1]), fw_pack(x[2], x[3]), fw_pack(x[4], x[5]),
                             fw_pack(x[6], x[7]));
            }
          }
          __syncwarp();  // the next tcgen05.ld needs the whole warp
        }
      } else if (lane == 0) {
        *failed = 1;
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*failed != 0 && threadIdx.x == 0) atomicExch(status, AYK_WAIT_TIMEOUT);
  if (warp == 4) {
    __syncwarp();
    tmem_dealloc(tmem_base, L::TMEM_COLS);
  }
}

template <int D, bool SAME>
int launch_wide(const void* q, int ld_q, const void* k_pages, const void* v_pages,
                const int* block_table, int table_stride, const int* row_start, const int* kv_len,
                void* out, int ld_out, int num_requests, int num_rows, int total_tiles,
                int num_heads, int num_kv_heads, int page_size, unsigned long long cache_rows,
                float scale, int window, int keep_first, const float* gate, int ld_gate,
                const float* sink, int* status, cudaStream_t stream) {
  using L = FwShape<D, SAME>;
  static const cudaError_t configured =
      cudaFuncSetAttribute(attention_prefill_wide_kernel<D, SAME>,
                           cudaFuncAttributeMaxDynamicSharedMemorySize, L::DYNAMIC);
  if (configured != cudaSuccess) return (int)configured;
  const int box_rows = page_size < FW_BN ? page_size : FW_BN;
  CUtensorMap map_q, map_k, map_v;
  int r = make_map_bf16_k64(&map_q, q, num_rows, (uint64_t)num_heads * D, ld_q, FW_BM);
  if (r == AYK_OK) r = make_map_bf16_k64(&map_k, k_pages, cache_rows, D, D, box_rows);
  if (r == AYK_OK) r = make_map_bf16_k64(&map_v, v_pages, cache_rows, D, D, box_rows);
  if (r != AYK_OK) return r;
  int page_shift = 0;
  while ((1 << page_shift) < page_size) ++page_shift;
  return launch_kernel(attention_prefill_wide_kernel<D, SAME>, dim3(num_heads, total_tiles),
                       dim3(FW_THREADS), L::DYNAMIC, stream, 1, map_q, map_k, map_v, box_rows,
                       block_table, table_stride, row_start, kv_len, (__nv_bfloat16*)out, ld_out,
                       num_requests, num_kv_heads, num_heads / num_kv_heads, page_size, page_shift,
                       scale, window, keep_first, total_tiles, gate, ld_gate, sink, status);
}

}  // namespace ayk

AYK_API void ayk_set_pdl(int on) { ayk::pdl_enabled() = on; }

// Query rows per CTA: the caller sizes the grid with it.
AYK_API int ayk_attention_prefill_wide_rows() { return ayk::FW_BM; }

// bfloat16. q: num_rows rows; `total_tiles` = sum over requests of ceil(rows / 128). Returns
// AYK_NOT_TAKEN, having run nothing, for what this kernel does not serve: head sizes other than 64
// and 128 (256 where the value pages are the key pages), pages whose slots are no power of two from 8
// up, a scale that is not positive, operands whose rows are not whole aligned 16-byte pieces.
AYK_API int ayk_attention_prefill_wide(const void* q, int ld_q, const void* k_pages,
                                       const void* v_pages, const int* block_table,
                                       int table_stride, const int* row_start, const int* kv_len,
                                       void* out, int ld_out, int num_requests, int num_rows,
                                       int total_tiles, int num_heads, int num_kv_heads,
                                       int head_dim, int page_size, int num_pages, float scale,
                                       int window, int keep_first, const float* gate, int ld_gate,
                                       const float* sink, int* status, void* stream) {
  using namespace ayk;
  if (num_requests == 0 || total_tiles == 0) return AYK_OK;
  if (num_requests < 0 || num_rows < 1 || total_tiles < 0 || num_heads < 1 || num_kv_heads < 1 ||
      num_heads % num_kv_heads || page_size < 1 || num_pages < 1 || table_stride < 1 || window < 0 ||
      keep_first < 0 || status == nullptr || (gate != nullptr && ld_gate < num_heads * head_dim)) {
    return AYK_BAD_ARGUMENT;
  }
  if (total_tiles > 65535) return AYK_TOO_LARGE;
  const bool same = k_pages == v_pages;
  const unsigned long long cache_rows = (unsigned long long)num_pages * num_kv_heads * page_size;
  if (!(scale > 0.f) || page_size < 8 || (page_size & (page_size - 1)) || cache_rows >= 2147483648ull ||
      ((uintptr_t)q % 16) || ((uintptr_t)out % 16) || ((uintptr_t)k_pages % 16) ||
      ((uintptr_t)v_pages % 16) || (ld_q % 8) || (ld_out % 8) || ((uintptr_t)gate % 16) ||
      (gate != nullptr && ld_gate % 4)) {
    return AYK_NOT_TAKEN;
  }
#define AYK_WIDE(D, SAME)                                                                          \
  return launch_wide<D, SAME>(q, ld_q, k_pages, v_pages, block_table, table_stride, row_start,     \
                              kv_len, out, ld_out, num_requests, num_rows, total_tiles, num_heads, \
                              num_kv_heads, page_size, cache_rows, scale, window, keep_first,      \
                              gate, ld_gate, sink, status, (cudaStream_t)stream)
  if (head_dim == 64 && !same) AYK_WIDE(64, false);
  if (head_dim == 128 && !same) AYK_WIDE(128, false);
  if (head_dim == 256 && same) AYK_WIDE(256, true);
#undef AYK_WIDE
  return AYK_NOT_TAKEN;
}
