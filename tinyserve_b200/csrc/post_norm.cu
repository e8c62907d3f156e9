// Residual sum with a norm on the sub-layer's output, fused with the norm in front of the next
// sub-layer. For a row x of the 32-bit stream and the pending sub-layer output d (model dtype):
//
//   y   = d / sqrt(mean(d^2) + eps_post) * gain(post_weight) * layer_scale * m  (when a post norm is pending;
//                                                                                  m a constant multiplier)
//   y   = (d + bias) * m * layer_scale                                           (without a post norm: a constant and
//                                                                                  a layer scale, with the sub-layer's
//                                                                                  output bias, if any)
//   x  <- x + y + s d2 + rows + vec                                               (written back unless `rows`; d2 the
//                                                                                  output of a sub-layer side by side with
//                                                                                  d and its constant, rows 32-bit and vec
//                                                                                  one value per column; each if given)
//   out = x / sqrt(mean(x^2) + eps) * gain(weight)
//
// gain(w) = 1 + w when the weight is stored around zero (`unit_offset`), else w. Everything is
// 32-bit; `out` is rounded once to the model dtype. Without a post norm y = d (the plain residual
// sum), so the kernel is also the norm with an offset weight alone. With `rows` only those rows
// are read, `out` has one row per entry and the stream is left as it is.
#define TS_PDL_CLASS PDL_ELEMENTWISE
#include "common.cuh"

namespace ts {

struct PostNormArgs {
  float* resid;
  const void* delta;        // may be null: nothing pending
  const void* post_weight;  // may be null: the pending output is added as it is
  const void* layer_scale;  // may be null
  const void* delta_bias;   // may be null: one value per column added to the pending output (only without a post norm)
  const void* weight;
  void* out;
  const int* rows;
  const void* second;       // may be null: a second pending output, model dtype, times second_scale
  const float* add_rows;    // may be null: 32-bit rows added to the stream
  const void* add_vec;      // may be null: one value per column added to the stream
  int num_rows, hidden;
  float second_scale;
  float post_eps, eps;
  float post_mult;          // a constant on the normed pending output
  int post_offset, offset;  // 1: the gain is 1 + weight
};

// Rows whose four neighbouring elements lie in one access: a CTA takes a row, a thread NV times 4 of its elements, which stay
// in registers throughout. Bound by latency (a few rows between two products), so what no kernel before this one writes
// (the weights) is asked for in front of the wait, all that belongs to the row at once behind it, and each of the two sums
// meets at one barrier. Needs hidden % 4 == 0 and hidden <= 4,096 (beyond, the registers do not hold a row). The kernel below /
// this one, rows of 1,024, bf16, both norms, back to back: 1 row 2.54 / 2.03 us, 64 2.84 / 2.11, 190 4.44 / 2.62, 500 5.15 / 3.04; from 1,000
// rows on equal. So it takes up to 511 rows of up to 1,024 values; longer ones as many as run at once, two CTAs an SM up to 2,560
// values, one beyond (registers): 4,096 values, 148 rows 4.1 / 3.7 us, 149 4.5 / 6.1, 511 7.0 / 11.6; 2,560 values, 296 rows 4.3 / 3.7, 297
// 5.3 / 5.8, 511 5.7 / 6.7.
static int post_row_most(int hidden) { return hidden <= 1024 ? 511 : hidden <= 2560 ? 2 * 148 : hidden <= 4096 ? 148 : 0; }
template <typename T, int NV>
__global__ void __launch_bounds__(512) post_norm_row_kernel(PostNormArgs a) {
  __shared__ float parts[2][32];
  pdl_trigger();
  const int hidden = a.hidden, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const bool normed = a.delta && a.post_weight;
  float gain[NV][4], scale[NV][4], w[NV][4], more[NV][4];       // of the post norm; layer scale; of the norm; added to the stream
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int i = (threadIdx.x + j * blockDim.x) * 4;
#pragma unroll
    for (int e = 0; e < 4; ++e) { gain[j][e] = 0.f; scale[j][e] = 1.f; w[j][e] = more[j][e] = 0.f; }
    if (i >= hidden) continue;
    if (normed) Quad<T>::load((const T*)a.post_weight + i, gain[j]);
    else if (a.delta_bias) Quad<T>::load((const T*)a.delta_bias + i, gain[j]);       // (in its place)
    if (a.layer_scale) Quad<T>::load((const T*)a.layer_scale + i, scale[j]);
    Quad<T>::load((const T*)a.weight + i, w[j]);
  }
  pdl_wait();
  const int r = blockIdx.x;
  const int row = a.rows ? a.rows[r] : r;
  float* x = a.resid + (size_t)row * hidden;
  const T* d = a.delta ? (const T*)a.delta + (size_t)row * hidden : nullptr;
  const T* d2 = a.second ? (const T*)a.second + (size_t)row * hidden : nullptr;
  const float* ar = a.add_rows ? a.add_rows + (size_t)row * hidden : nullptr;
  const bool write_back = (a.rows == nullptr) && (d != nullptr || ar != nullptr || a.add_vec != nullptr);
  float v[NV][4], y[NV][4], beside[NV][4], rows[NV][4];
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int i = (threadIdx.x + j * blockDim.x) * 4;
#pragma unroll
    for (int e = 0; e < 4; ++e) v[j][e] = y[j][e] = beside[j][e] = rows[j][e] = 0.f;
    if (i >= hidden) continue;
    if (d) Quad<T>::load(d + i, y[j]);
    Quad<float>::load(x + i, v[j]);
    if (d2) Quad<T>::load(d2 + i, beside[j]);
    if (ar) Quad<float>::load(ar + i, rows[j]);
    if (a.add_vec) Quad<T>::load((const T*)a.add_vec + i, more[j]);
  }
  auto row_sum = [&](float s, float* of) {
    s = warp_sum(s);
    if (lane == 0) of[threadIdx.x >> 5] = s;
    __syncthreads();
    return warp_sum(lane < warps ? of[lane] : 0.f);
  };
  float post_rstd = 1.f;
  if (normed) {
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) ss = fmaf(y[j][e], y[j][e], ss);
    post_rstd = rsqrtf(row_sum(ss, parts[0]) / (float)hidden + a.post_eps);
  }
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int i = (threadIdx.x + j * blockDim.x) * 4;
    if (i >= hidden) continue;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (d) {
        float t = normed ? y[j][e] * post_rstd * (a.post_offset ? 1.f + gain[j][e] : gain[j][e]) : a.delta_bias ? y[j][e] + gain[j][e] : y[j][e];
        t *= a.post_mult;
        if (a.layer_scale) t *= scale[j][e];
        v[j][e] += t;
        if (d2) v[j][e] = fmaf(a.second_scale, beside[j][e], v[j][e]);
      }
      if (ar) v[j][e] += rows[j][e];
      if (a.add_vec) v[j][e] += more[j][e];
      ss = fmaf(v[j][e], v[j][e], ss);
    }
    if (write_back) Quad<float>::store(x + i, v[j]);
  }
  const float rstd = rsqrtf(row_sum(ss, parts[1]) / (float)hidden + a.eps);
  T* o = (T*)a.out + (size_t)r * hidden;
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int i = (threadIdx.x + j * blockDim.x) * 4;
    if (i >= hidden) continue;
    float res[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) res[e] = v[j][e] * rstd * (a.offset ? 1.f + w[j][e] : w[j][e]);
    Quad<T>::store(o + i, res);
  }
}

// Other rows: the row lives in shared memory (32-bit) between the passes. VEC: 4 elements per
// access (needs hidden % 4 == 0 and 16-byte aligned rows), else 1.
template <typename T, int VEC>
__global__ void post_norm_add_rms_norm_kernel(PostNormArgs a) {
  extern __shared__ float xs[];
  __shared__ float scratch[33];
  pdl_trigger();
  pdl_wait();
  const int r = blockIdx.x, hidden = a.hidden;
  const int row = a.rows ? a.rows[r] : r;
  float* x = a.resid + (size_t)row * hidden;
  const T* d = a.delta ? (const T*)a.delta + (size_t)row * hidden : nullptr;
  const T* pw = (const T*)a.post_weight;
  const T* ls = (const T*)a.layer_scale;
  const T* db = (const T*)a.delta_bias;
  const T* w = (const T*)a.weight;
  const T* d2 = a.second ? (const T*)a.second + (size_t)row * hidden : nullptr;
  const float* ar = a.add_rows ? a.add_rows + (size_t)row * hidden : nullptr;
  const T* av = (const T*)a.add_vec;
  const bool write_back = (a.rows == nullptr) && (d != nullptr || ar != nullptr || av != nullptr);
  float post_rstd = 1.f;
  if (d && pw) {
    float ss = 0.f;
    for (int i = threadIdx.x * VEC; i < hidden; i += blockDim.x * VEC) {
      float f[VEC];
      if constexpr (VEC == 4) Quad<T>::load(d + i, f); else f[0] = to_float(d[i]);
#pragma unroll
      for (int e = 0; e < VEC; ++e) { xs[i + e] = f[e]; ss = fmaf(f[e], f[e], ss); }
    }
    ss = block_sum(ss, scratch);
    post_rstd = rsqrtf(ss / (float)hidden + a.post_eps);
  }
  float ss = 0.f;
  for (int i = threadIdx.x * VEC; i < hidden; i += blockDim.x * VEC) {
    float v[VEC];
    if constexpr (VEC == 4) Quad<float>::load(x + i, v); else v[0] = x[i];
    if (d) {
      float y[VEC];
      if (pw) {
        float g[VEC];
        if constexpr (VEC == 4) Quad<T>::load(pw + i, g); else g[0] = to_float(pw[i]);
#pragma unroll
        for (int e = 0; e < VEC; ++e) y[e] = xs[i + e] * post_rstd * (a.post_offset ? 1.f + g[e] : g[e]) * a.post_mult;
      } else {
        if constexpr (VEC == 4) Quad<T>::load(d + i, y); else y[0] = to_float(d[i]);
        if (db) {
          float b[VEC];
          if constexpr (VEC == 4) Quad<T>::load(db + i, b); else b[0] = to_float(db[i]);
#pragma unroll
          for (int e = 0; e < VEC; ++e) y[e] += b[e];
        }
#pragma unroll
        for (int e = 0; e < VEC; ++e) y[e] *= a.post_mult;
      }
      if (ls) {
        float s[VEC];
        if constexpr (VEC == 4) Quad<T>::load(ls + i, s); else s[0] = to_float(ls[i]);
#pragma unroll
        for (int e = 0; e < VEC; ++e) y[e] *= s[e];
      }
#pragma unroll
      for (int e = 0; e < VEC; ++e) v[e] += y[e];
      if (d2) {
        if constexpr (VEC == 4) Quad<T>::load(d2 + i, y); else y[0] = to_float(d2[i]);
#pragma unroll
        for (int e = 0; e < VEC; ++e) v[e] = fmaf(a.second_scale, y[e], v[e]);
      }
    }
    if (ar) {
      float y[VEC];
      if constexpr (VEC == 4) Quad<float>::load(ar + i, y); else y[0] = ar[i];
#pragma unroll
      for (int e = 0; e < VEC; ++e) v[e] += y[e];
    }
    if (av) {
      float y[VEC];
      if constexpr (VEC == 4) Quad<T>::load(av + i, y); else y[0] = to_float(av[i]);
#pragma unroll
      for (int e = 0; e < VEC; ++e) v[e] += y[e];
    }
    if (write_back) {
      if constexpr (VEC == 4) Quad<float>::store(x + i, v); else x[i] = v[0];
    }
#pragma unroll
    for (int e = 0; e < VEC; ++e) { xs[i + e] = v[e]; ss = fmaf(v[e], v[e], ss); }
  }
  ss = block_sum(ss, scratch);
  const float rstd = rsqrtf(ss / (float)hidden + a.eps);
  T* o = (T*)a.out + (size_t)r * hidden;
  for (int i = threadIdx.x * VEC; i < hidden; i += blockDim.x * VEC) {
    float g[VEC], res[VEC];
    if constexpr (VEC == 4) Quad<T>::load(w + i, g); else g[0] = to_float(w[i]);
#pragma unroll
    for (int e = 0; e < VEC; ++e) res[e] = xs[i + e] * rstd * (a.offset ? 1.f + g[e] : g[e]);
    if constexpr (VEC == 4) Quad<T>::store(o + i, res); else o[i] = from_float<T>(res[0]);
  }
}

}  // namespace ts

using namespace ts;

extern "C" int ts_post_norm_add_rms_norm(float* resid, const void* delta, const void* post_weight, const void* layer_scale,
                                         float post_eps, int post_offset, float post_mult, const void* weight, int offset,
                                         float eps, void* out, const int* rows, int num_rows, int hidden, const void* delta_bias,
                                         const void* second, float second_scale, const float* add_rows, const void* add_vec,
                                         int dtype, cudaStream_t stream) {
  if (num_rows <= 0) return 0;
  if (hidden <= 0 || hidden > 12288 || !weight || !out || !resid) return TS_ERR_BAD_ARGUMENT;
  if (dtype != TS_DTYPE_F32 && dtype != TS_DTYPE_BF16) return TS_ERR_BAD_ARGUMENT;
  if ((post_weight || layer_scale || delta_bias || second) && !delta) return TS_ERR_BAD_ARGUMENT;
  if (delta_bias && post_weight) return TS_ERR_UNSUPPORTED;
  PostNormArgs a;
  a.resid = resid; a.delta = delta; a.post_weight = post_weight; a.layer_scale = layer_scale; a.delta_bias = delta_bias; a.weight = weight;
  a.out = out; a.rows = rows; a.num_rows = num_rows; a.hidden = hidden; a.post_eps = post_eps; a.eps = eps;
  a.post_offset = post_offset; a.offset = offset; a.post_mult = post_mult;
  a.second = second; a.second_scale = second_scale; a.add_rows = add_rows; a.add_vec = add_vec;
  const size_t smem = sizeof(float) * (size_t)hidden;
  const bool aligned = hidden % 4 == 0 &&
      (((uintptr_t)resid | (uintptr_t)delta | (uintptr_t)post_weight | (uintptr_t)layer_scale | (uintptr_t)delta_bias | (uintptr_t)weight | (uintptr_t)out |
        (uintptr_t)second | (uintptr_t)add_rows | (uintptr_t)add_vec) & 15) == 0;
  if (aligned && num_rows <= post_row_most(hidden)) {
    const int quads = hidden / 4, threads = ((quads <= 512 ? quads : (quads + 1) / 2) + 31) / 32 * 32;
#define TS_PN_ROW(T_)                                                                          \
  return quads <= 512 ? launch(post_norm_row_kernel<T_, 1>, num_rows, threads, 0, stream, a)  \
                      : launch(post_norm_row_kernel<T_, 2>, num_rows, threads, 0, stream, a)
    if (dtype == TS_DTYPE_F32) TS_PN_ROW(float);
    TS_PN_ROW(bf16);
#undef TS_PN_ROW
  }
  const int per = aligned ? 4 : 1;
  int threads = 64;
  while (threads < 512 && threads * per * 2 <= hidden) threads <<= 1;
#define TS_PN_CASE(T_, V_)                                                                          \
  do {                                                                                              \
    auto kern = post_norm_add_rms_norm_kernel<T_, V_>;                                              \
    if (smem > 48 * 1024) {                                                                         \
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
      if (e != cudaSuccess) return (int)e;                                                          \
    }                                                                                               \
    return launch(kern, num_rows, threads, smem, stream, a);                                        \
  } while (0)
  if (dtype == TS_DTYPE_F32) { if (aligned) TS_PN_CASE(float, 4); TS_PN_CASE(float, 1); }
  if (aligned) TS_PN_CASE(bf16, 4);
  TS_PN_CASE(bf16, 1);
#undef TS_PN_CASE
}
