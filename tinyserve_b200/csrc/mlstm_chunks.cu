// The mLSTM recurrence (recurrent_scan.cu) for long prompt portions, as products over chunks of 64 tokens. With the log gates
// i_t and f_t, F_t the running sum of f within a chunk, g_s = i_s - F_s and R_t = max(m_0, max over s <= t of g_s), a chunk that
// starts from the state (S_0, n_0, m_0) has m_t = F_t + R_t and
//
//   S_t q_t = e^(m_0 - R_t) S_0^T q_t + sum_{s <= t} e^(g_s - R_t) (k_s . q_t) v_s           (n_t . q_t: the same with v = 1)
//   o_t     = S_t q_t / (max(|n_t . q_t|, e^(-m_t)) + 1e-6)
//   S'      = e^(F_end + m_0 - m') S_0 + e^(F_end - m') sum_s e^(g_s) k_s v_s^T,   m' = F_end + R_end      (n' likewise)
//
// the recurrence's own stabiliser, so every exponent but that of e^(-m_t) is at most zero.
//  * leave kernel   : the last sums of a chunk, in the scale of its largest g, and F_end and that g;
//  * combine kernel : walks a request's chunks in order, leaves each one's starting state in the place of those sums, and
//                     stores the request's slot;
//  * read kernel    : the scores of a chunk, weighted, times v plus q times S_0, over the normaliser.
//
// Token by token a step of the chain is some 700 cycles (read-outs of shared memory, which a thread spends on two
// multiply-adds each): a portion of 650 tokens of 8 heads of 128 took 240 us a layer; over chunks nothing but the combination
// of the chunks is a chain. 32-bit throughout on CUDA cores, as the state has to be; the running sums and what is
// subtracted from them in 64-bit, because a long or fast decaying chunk would lose the digits of their differences.
#define TS_PDL_CLASS PDL_OTHER
#include <cuda_pipeline_primitives.h>

#include "common.cuh"
#include "scan_chunks.cuh"

namespace ts {

struct MlstmChunkArgs {
  const void* qkv; int stride, q_off, k_off, v_off;     // [T, stride]
  const float* gates;                 // [T, 2 H] pre-activations: input, forget
  const float* gate_bias;             // [2 H]
  float cap, q_scale;
  float* state; int state_stride;     // per head: S [d][dv], then a copy of (n [d], m) per block of 32 value columns
  const int* cu_q; const int* state_slots;
  int num_seqs, H, d, dv;
  int h0, some;                       // the heads of this pass: h0 .. h0 + some (all, where the scratch holds all)
  float* out;                         // [T, H, dv]
  float* left;                        // [chunks, some, d, dv]: what a chunk leaves, then its starting state
  float* left_n;                      // [chunks, some, d]: the same of the normaliser
  double* ends;                       // [chunks, some, 2]: F_end and the largest g
  float* starts;                      // [chunks, some]: m_0
};

// e^x of a difference of sums in 64-bit: rounded to 32 bits, an x in the tens would leave its last digits to the result.
__device__ __forceinline__ float exp_of(double x) {
  const float hi = (float)x, e = expf(hi);
  // (below -100 both are zero, and x may be -inf; e^(-m) may be more than 32 bits hold)
  return hi > -100.f && e < INFINITY ? fmaf(e, (float)(x - (double)hi), e) : e;
}

// By one warp: F and g of the chunk's tokens (two a lane; past the end F stays and g is -inf), and the largest g so far.
__device__ __forceinline__ void mlstm_gates(const MlstmChunkArgs& a, int h, int t0, int nt, int lane, double* cum_s, double* g_s, double* top_s) {
  const float bi = a.gate_bias[h], bf = a.gate_bias[a.H + h];
  float li[2];
  double lf[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int t = 2 * lane + i;
    li[i] = -INFINITY;
    lf[i] = 0.0;
    if (t < nt) {
      const float* z = a.gates + (size_t)(t0 + t) * 2 * a.H;
      li[i] = a.cap * tanhf((z[h] + bi) / a.cap);
      const float f = a.cap * tanhf((z[a.H + h] + bf) / a.cap);
      lf[i] = f < 0.f ? f - log1pf(expf(f)) : -log1pf(expf(-f));
    }
  }
  double run = lf[0] + lf[1];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double other = __shfl_up_sync(0xffffffffu, run, o);
    if (lane >= o) run += other;
  }
  // (not run - lf[1]: a token whose gate is no number is not to be seen by the one before it)
  const double in_front = __shfl_up_sync(0xffffffffu, run, 1), f0 = (lane ? in_front : 0.0) + lf[0], f1 = run;
  const double g0 = (double)li[0] - f0, g1 = (double)li[1] - f1;
  double top = fmax(g0, g1);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double other = __shfl_up_sync(0xffffffffu, top, o);
    if (lane >= o) top = fmax(top, other);
  }
  const double before = __shfl_up_sync(0xffffffffu, top, 1);
  cum_s[2 * lane] = f0;
  cum_s[2 * lane + 1] = f1;
  g_s[2 * lane] = g0;
  g_s[2 * lane + 1] = g1;
  top_s[2 * lane] = lane ? fmax(before, g0) : g0;
  top_s[2 * lane + 1] = top;
}

// What a chunk leaves per head, [d x dv] and [d]. A CTA is (chunk, head, 64 value columns); NP = the key size rounded up to 64.
template <typename T, int NP>
__global__ void __launch_bounds__(2 * NP) mlstm_leave_kernel(MlstmChunkArgs a) {
  constexpr int THREADS = 2 * NP;     // (NP / 8) x (64 / 4) tiles of 8 x 4
  extern __shared__ __align__(16) float sc_smem[];
  float* k_s = sc_smem;               // [SC_Q][NP]
  float* v_s = k_s + SC_Q * NP;       // [SC_Q][SC_V], weighted
  __shared__ double cum_s[SC_Q], g_s[SC_Q], top_s[SC_Q];
  __shared__ float w_s[SC_Q];
  pdl_trigger();
  pdl_wait();
  int t0, nt;
  const int g = blockIdx.x, h = a.h0 + blockIdx.y, v0 = blockIdx.z * SC_V;
  if (!find_chunk(a.cu_q, a.num_seqs, g, t0, nt)) return;
  const int tid = threadIdx.x, lane = tid & 31;
  if (tid < 32) mlstm_gates(a, h, t0, nt, lane, cum_s, g_s, top_s);
  const T* kp = (const T*)a.qkv + (size_t)t0 * a.stride + a.k_off + h * a.d;
  const T* vp = (const T*)a.qkv + (size_t)t0 * a.stride + a.v_off + h * a.dv + v0;
  load_rows(vp, a.stride, nt, min(SC_V, a.dv - v0), rows_aligned(vp, a.stride), v_s, SC_V, SC_V, nt, tid, THREADS);
  load_rows(kp, a.stride, nt, a.d, rows_aligned(kp, a.stride), k_s, NP, NP, nt, tid, THREADS);
  __syncthreads();
  const double top = top_s[SC_Q - 1];
  if (tid < SC_Q) w_s[tid] = tid < nt ? exp_of(g_s[tid] - top) : 0.f;
  __syncthreads();
  for (int idx = tid; idx < nt * (SC_V / 4); idx += THREADS) {
    const float w = w_s[idx / (SC_V / 4)];
    float4* p = reinterpret_cast<float4*>(v_s) + idx;
    float4 v = *p;
    v.x *= w; v.y *= w; v.z *= w; v.w *= w;
    *p = v;
  }
  const size_t at = (size_t)g * a.some + blockIdx.y;
  if (blockIdx.z == 0) {
    if (tid == 0) {
      a.ends[2 * at] = cum_s[SC_Q - 1];
      a.ends[2 * at + 1] = top;
    }
    if (tid < a.d) {
      float n = 0.f;
      for (int t = 0; t < nt; ++t) n = fmaf(w_s[t], k_s[t * NP + tid], n);
      a.left_n[at * a.d + tid] = n;
    }
  }
  __syncthreads();
  const int n_at = (tid / 16) * 8, v_at = (tid % 16) * 4;
  float acc[8][4] = {};
  tile_product_in_blocks<2>(acc, k_s + n_at, NP, v_s + v_at, SC_V, nt);
  float* dst = a.left + at * a.d * a.dv + v0 + v_at;
  const bool vec = (a.dv & 3) == 0 && v0 + v_at + 4 <= a.dv;
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    if (n_at + r >= a.d) break;
    float* p = dst + (size_t)(n_at + r) * a.dv;
    if (vec) {
      *reinterpret_cast<float4*>(p) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (v0 + v_at + j < a.dv) p[j] = acc[r][j];
    }
  }
}

// A request's chunks in order. A thread per VEC elements of S; the last CTA of a head (blockIdx.z) has the normaliser.
constexpr int MC_AHEAD = 8;       // chunks whose loads are in flight
template <int VEC>
__global__ void __launch_bounds__(128) mlstm_combine_kernel(MlstmChunkArgs a) {
  pdl_trigger();
  pdl_wait();
  const int b = blockIdx.x, h = a.h0 + blockIdx.y;
  const int start = a.cu_q[b], n = a.cu_q[b + 1] - start;
  if (n <= 0) return;
  const int copies = (a.dv + 31) / 32, per_head = a.d * a.dv;
  const int chunks = (n + SC_Q - 1) / SC_Q, first = start / SC_Q + b;
  float* head = a.state + (size_t)a.state_slots[b] * a.state_stride + (size_t)h * ((size_t)per_head + (size_t)copies * (a.d + 1));
  float* of_n = head + per_head;
  const bool normaliser = blockIdx.z == gridDim.z - 1;
  const int idx = (normaliser ? threadIdx.x : blockIdx.z * blockDim.x + threadIdx.x) * VEC;
  const int size = normaliser ? a.d : per_head;
  const bool mine = idx < size;
  float* p0 = (normaliser ? a.left_n : a.left) + ((size_t)first * a.some + blockIdx.y) * size + idx;
  const size_t step = (size_t)a.some * size;
  double* e0 = a.ends + ((size_t)first * a.some + blockIdx.y) * 2;
  const size_t estep = (size_t)a.some * 2;
  float s[VEC], m = of_n[a.d];
#pragma unroll
  for (int e = 0; e < VEC; ++e) s[e] = mine && idx + e < size ? (normaliser ? of_n : head)[idx + e] : 0.f;
  for (int c0 = 0; c0 < chunks; c0 += MC_AHEAD) {
    float left[MC_AHEAD][VEC];
    double fall[MC_AHEAD], top[MC_AHEAD];
#pragma unroll
    for (int j = 0; j < MC_AHEAD; ++j) {
      const bool in = c0 + j < chunks;
      fall[j] = in ? e0[(c0 + j) * estep] : 0.0;
      top[j] = in ? e0[(c0 + j) * estep + 1] : 0.0;
#pragma unroll
      for (int e = 0; e < VEC; ++e) left[j][e] = 0.f;
      if (in && mine) {
        const float* p = p0 + (size_t)(c0 + j) * step;
        if constexpr (VEC == 4) Quad<float>::load(p, left[j]); else left[j][0] = p[0];
      }
    }
#pragma unroll
    for (int j = 0; j < MC_AHEAD; ++j) {
      if (c0 + j >= chunks) break;
      if (mine) {
        float* p = p0 + (size_t)(c0 + j) * step;
        if constexpr (VEC == 4) Quad<float>::store(p, s); else p[0] = s[0];
      }
      // (S and n carry e^(-m) with m as it is stored, rounded to 32 bits)
      const float m_new = (float)(fall[j] + fmax((double)m, top[j]));
      const float keep = exp_of(fall[j] + (double)m - (double)m_new), take = exp_of(fall[j] + top[j] - (double)m_new);
      if (normaliser && threadIdx.x == 0) a.starts[(size_t)(first + c0 + j) * a.some + blockIdx.y] = m;
#pragma unroll
      for (int e = 0; e < VEC; ++e) s[e] = fmaf(keep, s[e], take * left[j][e]);
      m = m_new;
    }
  }
  if (normaliser) {
    for (int c = 0; c < copies; ++c) {
      float* copy = of_n + (size_t)c * (a.d + 1);
#pragma unroll
      for (int e = 0; e < VEC; ++e)
        if (mine && idx + e < size) copy[idx + e] = s[e];       // (m itself is stored by the read kernel: others still read it)
    }
  } else if (mine) {
#pragma unroll
    for (int e = 0; e < VEC; ++e) head[idx + e] = s[e];
  }
}

// The read-outs of a chunk. A CTA is (chunk, head, 64 value columns).
constexpr int MC_THREADS = 256;       // (64 / 4) x (64 / 4) tiles of 4 x 4
template <typename T, int NP>
__global__ void __launch_bounds__(MC_THREADS, 2) mlstm_read_kernel(MlstmChunkArgs a) {
  extern __shared__ __align__(16) float sc_smem[];
  float* q_s = sc_smem;               // [NP][SC_LD]: q, token fastest
  float* s_s = q_s + NP * SC_LD;      // [NP][SC_LD]: k, token fastest; then [NP][SC_V]: the starting state
  float* v_s = s_s + NP * SC_LD;      // [SC_Q][SC_V]
  float* m_s = v_s + SC_Q * SC_V;     // [SC_Q][SC_LD]: weighted scores, row s, token t fastest
  __shared__ double cum_s[SC_Q], g_s[SC_Q], top_s[SC_Q];
  __shared__ float n_s[NP], fall_s[SC_Q], den_s[4][SC_Q];
  pdl_trigger();
  pdl_wait();
  int t0, nt, seq;
  const int g = blockIdx.x, h = a.h0 + blockIdx.y, v0 = blockIdx.z * SC_V, d = a.d;
  if (!find_chunk(a.cu_q, a.num_seqs, g, t0, nt, &seq)) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t at = (size_t)g * a.some + blockIdx.y;
  const T* row = (const T*)a.qkv + (size_t)t0 * a.stride;
  load_transposed(row + a.q_off + h * d, a.stride, nt, d, NP, q_s, warp, MC_THREADS / 32, lane, a.q_scale);
  load_transposed(row + a.k_off + h * d, a.stride, nt, d, NP, s_s, warp, MC_THREADS / 32, lane);
  const T* vp = row + a.v_off + h * a.dv + v0;
  const int cols = min(SC_V, a.dv - v0);
  load_rows(vp, a.stride, nt, cols, rows_aligned(vp, a.stride), v_s, SC_V, SC_V, SC_Q, tid, MC_THREADS);
  if (warp == 0) mlstm_gates(a, h, t0, nt, lane, cum_s, g_s, top_s);
  for (int i = tid; i < NP; i += MC_THREADS) n_s[i] = i < d ? a.left_n[at * d + i] : 0.f;
  const double m0 = (double)a.starts[at];
  __syncthreads();
  const int t_at = (tid / 16) * 4, col = (tid % 16) * 4;   // this thread's tokens; its keys s, or its value columns
  const bool live = t_at < nt;
  float score[4][4] = {};
  if (live && col <= t_at + 3) tile_product_in_blocks<1>(score, q_s + t_at, SC_LD, s_s + col, SC_LD, d);
  __syncthreads();                    // k has been read
  // the starting state travels while the weighted scores are made
  const float* sp = a.left + at * d * a.dv + v0;
  if (cols == SC_V && rows_aligned(sp, a.dv)) {
    for (int idx = tid; idx < d * (SC_V / 4); idx += MC_THREADS)
      __pipeline_memcpy_async(s_s + idx * 4, sp + (size_t)(idx / (SC_V / 4)) * a.dv + (idx % (SC_V / 4)) * 4, 16);
  } else {
    load_rows(sp, a.dv, d, cols, rows_aligned(sp, a.dv), s_s, SC_V, SC_V, d, tid, MC_THREADS);
  }
  __pipeline_commit();
  if (tid < SC_Q) fall_s[tid] = exp_of(m0 - fmax(m0, top_s[tid]));
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int s = col + j;
    float m[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int t = t_at + r;
      m[r] = s <= t && t < nt ? score[r][j] * exp_of(g_s[s] - fmax(m0, top_s[t])) : 0.f;
    }
    *reinterpret_cast<float4*>(m_s + s * SC_LD + t_at) = make_float4(m[0], m[1], m[2], m[3]);
  }
  __syncthreads();
  {
    // n_t . q_t, a quarter of its terms a thread
    const int t = tid & (SC_Q - 1), part = tid / SC_Q;
    float own = 0.f, before = 0.f;
    for (int s = part; s < nt; s += 4) own += m_s[s * SC_LD + t];
    for (int i = part; i < d; i += 4) before = fmaf(n_s[i], q_s[i * SC_LD + t], before);
    den_s[part][t] = fmaf(fall_s[t], before, own);
  }
  __pipeline_wait_prior(0);
  __syncthreads();
  if (live) {
    float acc[4][4] = {};
    tile_product_in_blocks<1>(acc, q_s + t_at, SC_LD, s_s + col, SC_V, d);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float f = fall_s[t_at + r];
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[r][j] *= f;
    }
    tile_product_in_blocks<1>(acc, m_s + t_at, SC_LD, v_s + col, SC_V, t_at);
    // the four keys that not all of the thread's tokens see: left out, not multiplied by zero (a value may be infinite)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int s = t_at + j;
      if (s >= nt) break;
      const float4 m = *reinterpret_cast<const float4*>(m_s + s * SC_LD + t_at), v = *reinterpret_cast<const float4*>(v_s + s * SC_V + col);
      const float mv[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
      for (int r = j; r < 4; ++r) {
        acc[r][0] = fmaf(mv[r], v.x, acc[r][0]);
        acc[r][1] = fmaf(mv[r], v.y, acc[r][1]);
        acc[r][2] = fmaf(mv[r], v.z, acc[r][2]);
        acc[r][3] = fmaf(mv[r], v.w, acc[r][3]);
      }
    }
    const bool vec = (a.dv & 3) == 0 && col + 4 <= cols;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int t = t_at + r;
      if (t >= nt) break;
      const float nq = (den_s[0][t] + den_s[1][t]) + (den_s[2][t] + den_s[3][t]);
      const float by = fmaxf(fabsf(nq), exp_of(-(cum_s[t] + fmax(m0, top_s[t])))) + 1e-6f;
      float* p = a.out + ((size_t)(t0 + t) * a.H + h) * a.dv + v0 + col;
      if (vec) {
        *reinterpret_cast<float4*>(p) = make_float4(acc[r][0] / by, acc[r][1] / by, acc[r][2] / by, acc[r][3] / by);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (col + j < cols) p[j] = acc[r][j] / by;
      }
    }
  }
  // the request's last chunk: m after it, beside every copy of the normaliser
  if (v0 == 0 && t0 + nt == a.cu_q[seq + 1]) {
    const int copies = (a.dv + 31) / 32;
    float* of_n = a.state + (size_t)a.state_slots[seq] * a.state_stride +
                  (size_t)h * ((size_t)d * a.dv + (size_t)copies * (d + 1)) + (size_t)d * a.dv;
    const float m = (float)(cum_s[SC_Q - 1] + fmax(m0, top_s[SC_Q - 1]));
    for (int c = tid; c < copies; c += MC_THREADS) of_n[(size_t)c * (d + 1) + d] = m;
  }
}

template <typename T, int NP>
static int launch_mlstm_chunks(MlstmChunkArgs a, int chunks, cudaStream_t stream) {
  const int vblocks = (a.dv + SC_V - 1) / SC_V, per_head = a.d * a.dv;
  const size_t leave = sizeof(float) * SC_Q * (NP + SC_V);
  const size_t read = sizeof(float) * (2 * (size_t)NP * SC_LD + SC_Q * SC_V + SC_Q * SC_LD);
  auto lk = mlstm_leave_kernel<T, NP>;
  auto rk = mlstm_read_kernel<T, NP>;
  if (int e = (int)cudaFuncSetAttribute(lk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)leave)) return e;
  if (int e = (int)cudaFuncSetAttribute(rk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)read)) return e;
  const int vec = a.d % 4 == 0 ? 4 : 1, most = a.some;
  for (; a.h0 < a.H; a.h0 += most) {       // (each kernel waits for the pass before, whose scratch it takes over)
    a.some = a.H - a.h0 < most ? a.H - a.h0 : most;
    if (int e = launch(lk, dim3(chunks, a.some, vblocks), 2 * NP, leave, stream, a)) return e;
    const dim3 cgrid(a.num_seqs, a.some, (per_head / vec + 127) / 128 + 1);
    if (int e = vec == 4 ? launch(mlstm_combine_kernel<4>, cgrid, 128, 0, stream, a) : launch(mlstm_combine_kernel<1>, cgrid, 128, 0, stream, a)) return e;
    if (int e = launch(rk, dim3(chunks, a.some, vblocks), MC_THREADS, read, stream, a)) return e;
  }
  return 0;
}

}  // namespace ts

using namespace ts;

// As ts_mlstm_scan, d up to 128, `some` heads at a time; left [chunks, some, d, dv], left_n [chunks, some, d], ends
// [chunks, some, 2] doubles and starts [chunks, some] are scratch with chunks = num_tokens / 64 + num_seqs.
extern "C" int ts_mlstm_chunks(const void* qkv, int stride, int q_off, int k_off, int v_off, const float* gates, const float* gate_bias,
                               float cap, float q_scale, float* state, int state_stride, const int* cu_q, const int* state_slots,
                               int num_seqs, int num_tokens, int heads, int some, int d, int dv, float* left, float* left_n, double* ends,
                               float* starts, float* out, int dtype, cudaStream_t stream) {
  if (num_seqs <= 0 || num_tokens <= 0) return 0;
  if (heads <= 0 || some <= 0 || some > heads || d <= 0 || dv <= 0 || !(cap > 0.f) || !left || !left_n || !ends || !starts || !state || !out) return TS_ERR_BAD_ARGUMENT;
  if (d > SC_MAX_STATE || (((uintptr_t)left | (uintptr_t)left_n | (uintptr_t)ends | (uintptr_t)out) & 15)) return TS_ERR_UNSUPPORTED;
  MlstmChunkArgs a;
  a.qkv = qkv; a.stride = stride; a.q_off = q_off; a.k_off = k_off; a.v_off = v_off;
  a.gates = gates; a.gate_bias = gate_bias; a.cap = cap; a.q_scale = q_scale; a.state = state; a.state_stride = state_stride;
  a.cu_q = cu_q; a.state_slots = state_slots; a.num_seqs = num_seqs; a.H = heads; a.d = d; a.dv = dv;
  a.h0 = 0; a.some = some; a.out = out; a.left = left; a.left_n = left_n; a.ends = ends; a.starts = starts;
  const int chunks = num_tokens / SC_Q + num_seqs;
  if (dtype == TS_DTYPE_F32) return d <= 64 ? launch_mlstm_chunks<float, 64>(a, chunks, stream) : launch_mlstm_chunks<float, 128>(a, chunks, stream);
  if (dtype == TS_DTYPE_BF16) return d <= 64 ? launch_mlstm_chunks<bf16, 64>(a, chunks, stream) : launch_mlstm_chunks<bf16, 128>(a, chunks, stream);
  return TS_ERR_BAD_ARGUMENT;
}
