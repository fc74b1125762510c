// The recurrences with one decay per head (Mamba-2, mLSTM) over prompt portions, in chunks of 64
// rows: S_t = g_t S_(t-1) + m_t k_t v_t^T, y_t = S_t^T q_t, with g_t in [0, 1]. Walked row by row
// the scan is bound by one row's latency and by fetching k and q for a fused multiply-add or two
// an entry; over a chunk both become small matrix products with register tiles:
//   states:  a CTA per head, request and 64 x 64 piece of S carries its piece in registers over the
//            rows, S <- G S + sum_j (m_j g_(j+1) ... g_end) k_j v_j^T in stages of 32 rows, and
//            leaves the S in front of every chunk in scratch;
//   outputs: a CTA per chunk, head and 64 columns, all at once: row i of the chunk is
//            y_i = G_i q_i S_0 + sum_(j<=i) (D_ij m_j (q_i . k_j)) v_j,  D_ij = g_(j+1) ... g_i,
//            and G_i = g_0 ... g_i.
// Decays only appear as products of factors in [0, 1], formed factor by factor (never as quotients
// or as differences of sums of logarithms), so nothing overflows or cancels; all of it is fp32 FMA.
// Bound by shared memory (12 to 16 bytes a lane per 8 to 16 FMAs) and FMA issue.
// Measured on a B200, 4,024 rows of 4 requests, the longest 1,300 (gates, states and outputs):
// Mamba-2, 32 heads of 128 x 64: 1,250 -> 290 microseconds; mLSTM, 4 heads of 256 x 256: 1,412 -> 290.
#pragma once

namespace ayk {

constexpr int MC_ROWS = 64;    // rows of a chunk
constexpr int MC_STAGE = 32;   // rows of a stage of the states' ring
constexpr int MC_STAGES = 5;
constexpr int MC_TILE = 64;    // n and p of a piece of S, columns of an output tile
constexpr int MC_SLAB = 32;    // n of a slab of the outputs
constexpr int MC_LDQ = MC_SLAB + 4, MC_LDA = MC_ROWS + 4;

struct MemoryArgs {
  const float* q;      // row 0: a group of `per` heads shares N entries
  const float* k;
  const float* v;      // row 0: heads x P
  const float* gates;  // [rows][heads] decays g, then as many m, then (mLSTM) the floors e^-m
  float* states;       // [chunk][head][N][P]
  float* norms;        // [chunk][head][N] (mLSTM), else null
  float* state;        // slots: S as [head][P][N], then (mLSTM) n as [head][tiles][N]
  const int* row_start;
  const int* state_slot;
  const float* skip;   // [heads] (Mamba-2) or null
  float* out;          // heads x P a row
  long long state_stride;
  int ld_q, ld_k, ld_v, ld_out, per, requests, heads, N, P, rows, tiles;
  float q_scale;
};

__device__ __forceinline__ int mc_chunks_before(const int* row_start, int b) {
  int before = 0;
  for (int i = 0; i < b; ++i) {
    before += (row_start[i + 1] - row_start[i] + MC_ROWS - 1) / MC_ROWS;
  }
  return before;
}
// 16 bytes from `src` where `in`, else zeros (nothing is read then)
__device__ __forceinline__ void mc_copy(float* dst, const float* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(in ? 16 : 0)
               : "memory");
}

// Mamba-2's factors of every row and head: g = exp(-exp(A_log) dt) and m = dt.
__global__ void mamba2_gates_kernel(const float* __restrict__ dt_raw, int ld_dt,
                                    const float* __restrict__ dt_bias,
                                    const float* __restrict__ a_log, float* __restrict__ gates,
                                    int rows, int heads) {
  pdl_launch_dependents();
  const int idx = blockIdx.x * blockDim.x + threadIdx.x, row = idx / heads, h = idx % heads;
  if (row >= rows) return;
  const float rate = -expf(a_log[h]), bias = dt_bias[h];
  pdl_wait_for(dt_raw, gates);
  const float dt = softplus_f(dt_raw[(size_t)row * ld_dt + h] + bias);
  gates[idx] = expf(rate * dt);
  gates[(size_t)rows * heads + idx] = dt;
}

// mLSTM's, a CTA per head and request: the running maximum by a scan over 512 rows at a time (row
// i maps m to max(f_i + m, i_i); two such maps compose to one of the same form), then
// g = e^(f + m - m'), m = e^(i - m') and the floor e^-m'.
constexpr int MC_GATE_THREADS = 512;
__global__ void __launch_bounds__(MC_GATE_THREADS)
mlstm_gates_kernel(const float* __restrict__ proj, int ld_proj, int i_offset, int f_offset,
                   const float* __restrict__ gate_bias, float cap, float* __restrict__ state,
                   long long state_stride, long long max_offset, int tiles,
                   const int* __restrict__ row_start, const int* __restrict__ state_slot,
                   float* __restrict__ gates, int rows, int heads) {
  __shared__ float a_s[MC_GATE_THREADS / 32], b_s[MC_GATE_THREADS / 32];
  __shared__ float end_m;
  pdl_launch_dependents();
  const int h = blockIdx.x, b = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r0 = row_start[b], count = row_start[b + 1] - r0;
  const float bias_i = gate_bias != nullptr ? gate_bias[h] : 0.f;
  const float bias_f = gate_bias != nullptr ? gate_bias[heads + h] : 0.f;
  if (state_slot[b] < 0 || count <= 0) return;
  float* kept = state + (size_t)state_slot[b] * state_stride + max_offset + (size_t)h * tiles;
  pdl_wait_for(proj, kept, gates);
  float m_run = *kept;
  const size_t plane = (size_t)rows * heads;
  for (int t0 = 0; t0 < count; t0 += MC_GATE_THREADS) {
    const int t = t0 + tid;
    const bool row = t < count;
    const float* from = proj + (size_t)(r0 + (row ? t : 0)) * ld_proj;
    const float ig = row ? cap * tanhf((from[i_offset + h] + bias_i) / cap) : 0.f;
    const float f = row ? log_sigmoid_f(cap * tanhf((from[f_offset + h] + bias_f) / cap)) : 0.f;
    float a = f, bmax = row ? ig : -INFINITY;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float a_up = __shfl_up_sync(0xffffffffu, a, o);
      const float b_up = __shfl_up_sync(0xffffffffu, bmax, o);
      if (lane >= o) {
        bmax = fmaxf(a + b_up, bmax);
        a += a_up;
      }
    }
    if (lane == 31) {
      a_s[warp] = a;
      b_s[warp] = bmax;
    }
    __syncthreads();
    float m_warp = m_run;  // the maximum in front of this warp's rows
    for (int w = 0; w < warp; ++w) m_warp = fmaxf(a_s[w] + m_warp, b_s[w]);
    const float m_new = fmaxf(a + m_warp, bmax);
    float m_old = __shfl_up_sync(0xffffffffu, m_new, 1);
    if (lane == 0) m_old = m_warp;
    if (row) {
      const size_t at = (size_t)(r0 + t) * heads + h;
      gates[at] = expf(f + m_old - m_new);
      gates[plane + at] = expf(ig - m_new);
      gates[2 * plane + at] = expf(-m_new);
    }
    if (t == min(count, t0 + MC_GATE_THREADS) - 1) end_m = m_new;
    __syncthreads();
    m_run = end_m;
  }
  for (int i = tid; i < tiles; i += MC_GATE_THREADS) kept[i] = m_run;
}

// grid (heads, requests, pieces of S): 128 threads, each 4 x 8 entries (n: 4 ty .. + 3, p: 4 tx and
// 32 + 4 tx .. + 3). (64 threads of 8 x 8 fetch less from shared memory per FMA, but leave a
// scheduler less than a warp: 134 microseconds where this takes 124, at the sizes above.)
constexpr int MC_STATE_THREADS = 128;
template <bool NORM>
__global__ void __launch_bounds__(MC_STATE_THREADS)
memory_states_kernel(const MemoryArgs a) {
  extern __shared__ __align__(16) float mc_smem[];
  constexpr int STAGE_FLOATS = 2 * MC_STAGE * MC_TILE + 2 * MC_STAGE;
  pdl_launch_dependents();
  const int N = a.N, P = a.P, h = blockIdx.x, b = blockIdx.y;
  const int pieces_p = (P + MC_TILE - 1) / MC_TILE;
  const int n0 = (int)(blockIdx.z / pieces_p) * MC_TILE, p0 = (int)(blockIdx.z % pieces_p) * MC_TILE;
  const int tid = threadIdx.x, lane = tid & 31, tx = tid & 7, ty = tid >> 3;
  const int r0 = a.row_start[b], rows = a.row_start[b + 1] - r0;
  const int slot = a.state_slot[b];
  if (slot < 0 || rows <= 0) return;
  const int before = mc_chunks_before(a.row_start, b);
  float* mine = a.state + (size_t)slot * a.state_stride + (size_t)h * N * P;
  float* norm_mine = a.state + (size_t)slot * a.state_stride + (size_t)a.heads * N * P +
                     (size_t)h * a.tiles * N;
  const float* k = a.k;
  const float* v = a.v;
  const float* gates = a.gates;
  pdl_wait_for(k, v, gates, mine, norm_mine);
  k += (size_t)r0 * a.ld_k + (size_t)(h / a.per) * N + n0;
  v += (size_t)r0 * a.ld_v + (size_t)h * P + p0;
  gates += (size_t)r0 * a.heads + h;
  const size_t plane = (size_t)a.rows * a.heads;
  const int stages = (rows + MC_STAGE - 1) / MC_STAGE;
  auto stage = [&](int s) {
    if (s < stages) {
      float* at = mc_smem + s % MC_STAGES * STAGE_FLOATS;
      const int t0 = s * MC_STAGE;
      for (int idx = tid; idx < MC_STAGE * (MC_TILE / 4); idx += MC_STATE_THREADS) {
        const int i = idx / (MC_TILE / 4), c = idx % (MC_TILE / 4) * 4;
        const bool row = t0 + i < rows, in_n = row && n0 + c < N, in_p = row && p0 + c < P;
        mc_copy(at + i * MC_TILE + c, in_n ? k + (size_t)(t0 + i) * a.ld_k + c : k, in_n);
        mc_copy(at + MC_STAGE * MC_TILE + i * MC_TILE + c,
                in_p ? v + (size_t)(t0 + i) * a.ld_v + c : v, in_p);
      }
      float* g = at + 2 * MC_STAGE * MC_TILE;  // decays, then m
      if (tid < 2 * MC_STAGE) {
        const int i = tid % MC_STAGE, which = tid / MC_STAGE;
        if (t0 + i < rows) {
          copy_async(g + tid, gates + which * plane + (size_t)(t0 + i) * a.heads, 1);
        } else {
          g[tid] = which ? 0.f : 1.f;
        }
      }
    }
    copy_commit();
  };
#pragma unroll
  for (int s = 0; s < MC_STAGES - 1; ++s) stage(s);
  float acc[4][8];
  float norm = 0.f;
  auto n_of = [&](int i) { return n0 + ty * 4 + i; };
  auto p_of = [&](int j) { return p0 + tx * 4 + (j & 3) + (j >> 2) * 32; };
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int n = n_of(i), p = p_of(j);
      acc[i][j] = n < N && p < P ? mine[(size_t)p * N + n] : 0.f;
    }
  if (NORM && p0 == 0 && tid < MC_TILE && n0 + tid < N) norm = norm_mine[n0 + tid];
  for (int s = 0; s < stages; ++s) {
    copy_wait<MC_STAGES - 2>();
    __syncthreads();  // stage s has landed, and everyone is done with stage s - 1
    stage(s + MC_STAGES - 1);
    if (s % (MC_ROWS / MC_STAGE) == 0) {  // a chunk begins: its S
      const size_t chunk = (size_t)(before + s / (MC_ROWS / MC_STAGE)) * a.heads + h;
      float* to = a.states + chunk * N * P;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int j = 0; j < 8; j += 4) {
          if (n_of(i) < N && p_of(j) < P) {
            *reinterpret_cast<float4*>(to + (size_t)n_of(i) * P + p_of(j)) =
                make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]);
          }
        }
      }
      if (NORM && p0 == 0 && tid < MC_TILE && n0 + tid < N) a.norms[chunk * N + n0 + tid] = norm;
    }
    const float* k_s = mc_smem + s % MC_STAGES * STAGE_FLOATS;
    const float* v_s = k_s + MC_STAGE * MC_TILE;
    const float* g_s = v_s + MC_STAGE * MC_TILE;
    // lane i: the product of the decays behind row i, and the whole stage's
    float after = lane + 1 < 32 ? g_s[lane + 1] : 1.f;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float down = __shfl_down_sync(0xffffffffu, after, o);
      if (lane + o < 32) after *= down;
    }
    const float whole = __shfl_sync(0xffffffffu, after * g_s[0], 0);
    const float weight = after * g_s[MC_STAGE + lane];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] *= whole;
    if (NORM) norm *= whole;
#pragma unroll 4
    for (int r = 0; r < MC_STAGE; ++r) {
      const float w = __shfl_sync(0xffffffffu, weight, r);
      const float4 k0 = *reinterpret_cast<const float4*>(k_s + r * MC_TILE + ty * 4);
      const float4 v0 = *reinterpret_cast<const float4*>(v_s + r * MC_TILE + tx * 4);
      const float4 v1 = *reinterpret_cast<const float4*>(v_s + r * MC_TILE + 32 + tx * 4);
      const float kv[4] = {w * k0.x, w * k0.y, w * k0.z, w * k0.w};
      const float vv[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(kv[i], vv[j], acc[i][j]);
      if (NORM && p0 == 0 && tid < MC_TILE) norm = fmaf(w, k_s[r * MC_TILE + tid], norm);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int n = n_of(i), p = p_of(j);
      if (n < N && p < P) mine[(size_t)p * N + n] = acc[i][j];
    }
  if (NORM && p0 == 0 && tid < MC_TILE && n0 + tid < N) {
    for (int t = 0; t < a.tiles; ++t) norm_mine[(size_t)t * N + n0 + tid] = norm;
  }
}

// Four products summed before they join a long sum: an addition more, and a quarter of the chain of
// roundings (the row by row scan's lanes hold short sums too).
__device__ __forceinline__ float dot4(const float (&a)[4], float x, float y, float z, float w) {
  return fmaf(a[3], w, fmaf(a[2], z, fmaf(a[1], y, a[0] * x)));
}

constexpr int MC_SLAB_FLOATS = 2 * MC_ROWS * MC_LDQ + MC_SLAB * MC_TILE;
constexpr int MC_OUT_FLOATS = 2 * MC_SLAB_FLOATS + MC_ROWS * MC_LDA + 6 * MC_ROWS;
static_assert(MC_SLAB_FLOATS >= MC_ROWS * MC_TILE, "the values fit a slab's buffer");

// grid (chunks, heads, tiles of 64 columns): 128 threads; a thread owns rows ty + 8 i of the chunk
// and columns 4 tx .. + 3 of the outputs, tx + 16 j of the chunk's own matrix. Bound by issue (73 %
// of all slots). Packed pairs (fma.rn.f32x2) of neighbouring n issue half as much, but with the
// short sums below they need twice the registers and were slower: 185 microseconds where this
// takes 155, at the sizes above.
template <bool NORM>
__global__ void __launch_bounds__(128)
memory_outputs_kernel(const MemoryArgs a) {
  extern __shared__ __align__(16) float mc_smem[];
  float* m_s = mc_smem + 2 * MC_SLAB_FLOATS;  // [64][LDA]: D_ij m_j, then the chunk's matrix
  float* g_s = m_s + MC_ROWS * MC_LDA;        // decays, m, G_i, the floors, two shares of n . q
  float* take_s = g_s + MC_ROWS;
  float* whole_s = take_s + MC_ROWS;
  float* floor_s = whole_s + MC_ROWS;
  float* dot_s = floor_s + MC_ROWS;
  pdl_launch_dependents();
  const int N = a.N, P = a.P, h = blockIdx.y, p0 = blockIdx.z * MC_TILE;
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  int b = 0, index = blockIdx.x, rows = 0, r0 = 0;
  for (; b < a.requests; ++b) {
    r0 = a.row_start[b];
    rows = a.row_start[b + 1] - r0;
    const int chunks = (rows + MC_ROWS - 1) / MC_ROWS;
    if (index < chunks) break;
    index -= chunks;
  }
  if (b == a.requests || a.state_slot[b] < 0) return;
  const int t0 = index * MC_ROWS, count = min(MC_ROWS, rows - t0);
  r0 += t0;
  const size_t chunk = (size_t)blockIdx.x * a.heads + h;
  const float* q = a.q;
  const float* k = a.k;
  const float* v = a.v;
  const float* gates = a.gates;
  const float* states = a.states;
  const float* norms = a.norms;
  float* out = a.out;
  pdl_wait_for(q, k, v, gates, states, norms, out);
  q += (size_t)r0 * a.ld_q + (size_t)(h / a.per) * N;
  k += (size_t)r0 * a.ld_k + (size_t)(h / a.per) * N;
  v += (size_t)r0 * a.ld_v + (size_t)h * P + p0;
  states += chunk * N * P + p0;
  const int slabs = (N + MC_SLAB - 1) / MC_SLAB;
  auto stage = [&](int s) {
    if (s < slabs) {
      float* at = mc_smem + (s & 1) * MC_SLAB_FLOATS;
      const int n0 = s * MC_SLAB;
      for (int idx = tid; idx < MC_ROWS * (MC_SLAB / 4); idx += 128) {
        const int i = idx / (MC_SLAB / 4), c = idx % (MC_SLAB / 4) * 4;
        const bool in = i < count && n0 + c < N;
        mc_copy(at + i * MC_LDQ + c, in ? q + (size_t)i * a.ld_q + n0 + c : q, in);
        mc_copy(at + MC_ROWS * MC_LDQ + i * MC_LDQ + c,
                in ? k + (size_t)i * a.ld_k + n0 + c : k, in);
      }
      for (int idx = tid; idx < MC_SLAB * (MC_TILE / 4); idx += 128) {
        const int n = idx / (MC_TILE / 4), c = idx % (MC_TILE / 4) * 4;
        const bool in = n0 + n < N && p0 + c < P;
        mc_copy(at + 2 * MC_ROWS * MC_LDQ + n * MC_TILE + c,
                in ? states + (size_t)(n0 + n) * P + c : states, in);
      }
    } else if (s == slabs) {  // behind the last slab the values, [64][64]
      float* at = mc_smem + (s & 1) * MC_SLAB_FLOATS;
      for (int idx = tid; idx < MC_ROWS * (MC_TILE / 4); idx += 128) {
        const int i = idx / (MC_TILE / 4), c = idx % (MC_TILE / 4) * 4;
        const bool in = i < count && p0 + c < P;
        mc_copy(at + i * MC_TILE + c, in ? v + (size_t)i * a.ld_v + c : v, in);
      }
    }
    copy_commit();
  };
  const float* v_s = mc_smem + (slabs & 1) * MC_SLAB_FLOATS;
  stage(0);
  if (tid < MC_ROWS) {
    const size_t plane = (size_t)a.rows * a.heads, at = (size_t)(r0 + tid) * a.heads + h;
    const bool row = tid < count;
    g_s[tid] = row ? gates[at] : 1.f;
    take_s[tid] = row ? gates[plane + at] : 0.f;
    if (NORM) floor_s[tid] = row ? gates[2 * plane + at] : 1.f;
  }
  __syncthreads();
  {  // D_ij m_j, half a column a thread from the top (zeros above the diagonal)
    const int j = tid & 63, first = tid >> 6 ? 32 : 0;
    const float take = take_s[j];
    float d = 1.f;
    for (int i = j + 1; i < first; ++i) d *= g_s[i];
    for (int i = first; i < first + 32; ++i) {
      if (i > j) d *= g_s[i];
      m_s[i * MC_LDA + j] = i >= j ? d * take : 0.f;
    }
    if (j == 0) {  // (column 0's products, times g_0, are the G_i)
      float g = g_s[0];
      for (int i = 1; i < first; ++i) g *= g_s[i];
      for (int i = first; i < first + 32; ++i) {
        if (i > 0) g *= g_s[i];
        whole_s[i] = g;
      }
    }
  }
  float own[8][4], o[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) own[i][j] = o[i][j] = 0.f;
  float dot = 0.f;  // NORM: this thread's half slabs of row tid / 2's n_0 . q
  for (int s = 0; s < slabs; ++s) {
    stage(s + 1);
    copy_wait<1>();
    __syncthreads();
    const float* q_s = mc_smem + (s & 1) * MC_SLAB_FLOATS;
    const float* k_s = q_s + MC_ROWS * MC_LDQ;
    const float* s_s = k_s + MC_ROWS * MC_LDQ;
#pragma unroll 2
    for (int n = 0; n < MC_SLAB; n += 4) {
      float4 qv[8], kv[4], sv[4];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        qv[i] = *reinterpret_cast<const float4*>(q_s + (ty + 8 * i) * MC_LDQ + n);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        kv[j] = *reinterpret_cast<const float4*>(k_s + (tx + 16 * j) * MC_LDQ + n);
        sv[j] = *reinterpret_cast<const float4*>(s_s + (n + j) * MC_TILE + tx * 4);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float qe[4] = {qv[i].x, qv[i].y, qv[i].z, qv[i].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          own[i][j] += dot4(qe, kv[j].x, kv[j].y, kv[j].z, kv[j].w);
        }
        o[i][0] += dot4(qe, sv[0].x, sv[1].x, sv[2].x, sv[3].x);
        o[i][1] += dot4(qe, sv[0].y, sv[1].y, sv[2].y, sv[3].y);
        o[i][2] += dot4(qe, sv[0].z, sv[1].z, sv[2].z, sv[3].z);
        o[i][3] += dot4(qe, sv[0].w, sv[1].w, sv[2].w, sv[3].w);
      }
    }
    if (NORM) {
      const int n_at = s * MC_SLAB + (tid & 1) * (MC_SLAB / 2);
      const float* row = q_s + (tid >> 1) * MC_LDQ + (tid & 1) * (MC_SLAB / 2);
#pragma unroll
      for (int n = 0; n < MC_SLAB / 2; ++n) {
        if (n_at + n < N) dot = fmaf(row[n], norms[chunk * N + n_at + n], dot);
      }
    }
    __syncthreads();  // the slab is staged again at the turn after next
  }
  copy_wait<0>();
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      // (a later row's entry stays the zero it is: its product may be no number)
      if (tx + 16 * j <= ty + 8 * i) m_s[(ty + 8 * i) * MC_LDA + tx + 16 * j] *= own[i][j];
    }
  if (NORM) dot_s[tid] = dot;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) o[i][j] *= whole_s[ty + 8 * i];
#pragma unroll 2
  for (int j = 0; j < MC_ROWS; j += 4) {
    float4 av[8], vv[4];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      av[i] = *reinterpret_cast<const float4*>(m_s + (ty + 8 * i) * MC_LDA + j);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      vv[e] = *reinterpret_cast<const float4*>(v_s + (j + e) * MC_TILE + tx * 4);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float ae[4] = {av[i].x, av[i].y, av[i].z, av[i].w};
      // rows j + 1 + seen .. of the chunk are later than this one: zero times what they hold would
      // not be zero for an infinity
      const int seen = ty + 8 * i - j;
      if (seen >= 3) {
        o[i][0] += dot4(ae, vv[0].x, vv[1].x, vv[2].x, vv[3].x);
        o[i][1] += dot4(ae, vv[0].y, vv[1].y, vv[2].y, vv[3].y);
        o[i][2] += dot4(ae, vv[0].z, vv[1].z, vv[2].z, vv[3].z);
        o[i][3] += dot4(ae, vv[0].w, vv[1].w, vv[2].w, vv[3].w);
      } else if (seen >= 0) {
        const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 v1 = seen >= 1 ? vv[1] : none, v2 = seen >= 2 ? vv[2] : none;
        o[i][0] += dot4(ae, vv[0].x, v1.x, v2.x, 0.f);
        o[i][1] += dot4(ae, vv[0].y, v1.y, v2.y, 0.f);
        o[i][2] += dot4(ae, vv[0].z, v1.z, v2.z, 0.f);
        o[i][3] += dot4(ae, vv[0].w, v1.w, v2.w, 0.f);
      }
    }
  }
  if (NORM) {  // the denominators: two threads a row
    const int i = tid >> 1, half = (tid & 1) * 32;
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
      const float4 m = *reinterpret_cast<const float4*>(m_s + i * MC_LDA + half + j);
      sum += (m.x + m.y) + (m.z + m.w);
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    const float nq = fmaf(whole_s[i], dot_s[2 * i] + dot_s[2 * i + 1], sum) * a.q_scale;
    __syncthreads();  // (every share of n . q has been read)
    if ((tid & 1) == 0) dot_s[i] = fmaxf(fabsf(nq), floor_s[i]) + 1e-6f;
    __syncthreads();
  }
  const float skip = a.skip != nullptr ? a.skip[h] : 0.f;
  if (p0 + tx * 4 >= P) return;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = ty + 8 * i;
    if (r >= count) continue;
    float4 y = make_float4(o[i][0], o[i][1], o[i][2], o[i][3]);
    if (NORM) {
      const float below = dot_s[r];
      y.x = y.x * a.q_scale / below;
      y.y = y.y * a.q_scale / below;
      y.z = y.z * a.q_scale / below;
      y.w = y.w * a.q_scale / below;
    } else {
      const float4 x = *reinterpret_cast<const float4*>(v_s + r * MC_TILE + tx * 4);
      y.x = fmaf(skip, x.x, y.x);
      y.y = fmaf(skip, x.y, y.y);
      y.z = fmaf(skip, x.z, y.z);
      y.w = fmaf(skip, x.w, y.w);
    }
    *reinterpret_cast<float4*>(out + (size_t)(r0 + r) * a.ld_out + (size_t)h * P + p0 + tx * 4) = y;
  }
}

// Whether the chunked kernels read these operands: 16-byte pieces of every row.
inline bool memory_takes(const MemoryArgs& a) {
  const auto aligned = [](const void* p) { return ((uintptr_t)p % 16) == 0; };
  return a.N % 4 == 0 && a.P % 4 == 0 && a.ld_q % 4 == 0 && a.ld_k % 4 == 0 && a.ld_v % 4 == 0 &&
         a.ld_out % 4 == 0 && aligned(a.q) && aligned(a.k) && aligned(a.v) && aligned(a.out) &&
         aligned(a.states);
}

// Whether the grids of the chunked kernels count the rows, heads and pieces of a state.
inline bool memory_counts(int rows, int heads, int N, int P) {
  return heads <= 65535 && (long long)rows * heads <= 0x7fffff00LL &&
         (long long)((N + MC_TILE - 1) / MC_TILE) * ((P + MC_TILE - 1) / MC_TILE) <= 65535;
}

template <bool NORM>
int launch_memory(const MemoryArgs& a, int chunks, cudaStream_t stream) {
  constexpr int STATES_BYTES = MC_STAGES * (2 * MC_STAGE * MC_TILE + 2 * MC_STAGE) * 4;
  static const cudaError_t configured = [] {
    const cudaError_t e = cudaFuncSetAttribute(
        memory_states_kernel<NORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, STATES_BYTES);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(memory_outputs_kernel<NORM>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, MC_OUT_FLOATS * 4);
  }();
  if (configured != cudaSuccess) return (int)configured;
  const int pieces_n = (a.N + MC_TILE - 1) / MC_TILE, pieces_p = (a.P + MC_TILE - 1) / MC_TILE;
  const int status = launch_kernel(memory_states_kernel<NORM>,
                                   dim3(a.heads, a.requests, pieces_n * pieces_p),
                                   dim3(MC_STATE_THREADS),
                                   STATES_BYTES, stream, 1, a);
  if (status != AYK_OK) return status;
  return launch_kernel(memory_outputs_kernel<NORM>, dim3(chunks, a.heads, pieces_p), dim3(128),
                       MC_OUT_FLOATS * 4, stream, 1, a);
}

}  // namespace ayk
