// out[M, N] = x[M, K] * w[N, K]^T, all 32-bit floats, on CUDA cores (no tensor cores, no reduced precision).
// Two kernels for two regimes, one order of summation. K % 4 == 0 and 16-byte aligned pointers.
//
// Order of the sums. K is cut into 16 equal parts (4 * ceil(K / 64) long; the last ones may be shorter or empty). A
// part is one chain of fused multiply-adds in index order; four neighbouring parts make a group, added left to right;
// the four groups are added left to right. Both kernels, every tile and every split keep that order bit for bit, so a
// row's result depends neither on M nor on the rows beside it. (One chain over all of K, which this replaces, has the
// larger error: 16 short chains and 15 additions against K dependent roundings.)
//
// A few rows (M <= 16): bound by the stream of the weights. A CTA takes 8 rows of w; thread = (row, part), the 16
// parts of a row side by side, so 128 threads add up 128 chains and 1,024 weight rows already give 128 CTAs. Slabs of
// 32 k per part (16 KB of w) come through a ring of cp.async stages, the first ones in front of the wait for the
// kernels before this one. Every weight is read from shared memory once for up to 8 rows of x; from three rows and
// 2,048 columns on a thread owns two weight rows, because a broadcast word of x costs the shared memory as much as a
// word of w (8 rows of the 151,936 x 1,024 head: 207 us with one, 165 us with two). Measured back to back on B200, one
// row, 64 x 64 tiles of all K before / now: 4,096 x 1,024 70 / 11 us, 1,024 x 3,072 205 / 8 us, the head 92 us (6.8 TB/s).
//
// More rows: bound by the multiply-adds and, below some hundred rows, by the latency of the chains. Register tiles of
// 4 x 4 outputs a thread, 32 x 64 a CTA, operands in shared memory as [row][32 k] read in 16-byte words (rows a thread
// owns lie a stride apart, so that eight neighbouring threads read eight different groups of banks), three cp.async
// stages. Where the tiles are too few for the machine, the four groups of K go to the four CTAs of a cluster, which leave
// their sums in shared memory; each then adds up its share of the tile through distributed shared memory. Where parts are
// no whole steps of 32 k, a step runs over their ends (a part of its own steps multiplied mostly zeros: 1,000 rows of
// 10,000 x 100 298 us, of 512 x 64 24 us). Measured, one kernel of 64 x 64 tiles for all sizes (which these replace) /
// now: 45 rows of 4,096 x 1,024 76 / 20 us, 64 rows of 1,024 x 3,072 221 / 24 us, 190 rows of 6,144 x 1,024 115 / 67 us,
// 1,000 rows of 10,000 x 100 86 / 80 us, of 512 x 64 6.7 / 6.8; many rows reach 38 TFLOP/s. Tiles of 64 x 64 and
// 128 x 128 (8 outputs a thread and side) were no faster at any of 1 to 600 rows: they leave too few warps on an SM.
#define TS_PDL_CLASS PDL_OTHER
#include <cooperative_groups.h>

#include "common.cuh"

namespace ts {
namespace cg = cooperative_groups;

__device__ __forceinline__ void f32_copy16(float* dst, const float* src, bool ok) {
  const unsigned int d = (unsigned int)__cvta_generic_to_shared(dst);
  const int n = ok ? 16 : 0;     // zero-filled beyond the matrix
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void f32_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void f32_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

constexpr int FP_PARTS = 16;
__host__ __device__ __forceinline__ int f32_part_length(int K) { return 4 * ((K + 63) / 64); }

// ------------------------------------------------------------------------------------------------- a few rows
constexpr int FR_THREADS = 128, FR_SLAB = 32, FR_STRIDE = FR_SLAB + 4, FR_STAGES = 4;

// MT rows of x; a thread owns R rows of w (8 R a CTA).
template <int MT, int R>
struct F32Rows {
  static constexpr int ROWS = 8 * R;
  static constexpr int STAGE = FP_PARTS * ROWS * FR_STRIDE + MT * FP_PARTS * FR_SLAB;     // floats
};

// SHORT: a part is shorter than a slab.
template <int MT, int R, bool SHORT>
__global__ void __launch_bounds__(FR_THREADS) gemm_f32_rows_kernel(const float* x, const float* __restrict__ w, float* out,
                                                                  int M, int N, int K) {
  using Rows = F32Rows<MT, R>;
  constexpr int ROWS = Rows::ROWS;
  extern __shared__ float smem[];
  __shared__ float sums[4][ROWS][MT];
  pdl_trigger();
  const int tid = threadIdx.x, lane = tid & 31;
  const int row = lane & 7, part = (tid >> 5) * 4 + (lane >> 3);     // a warp holds one group of four parts
  const int n0 = blockIdx.x * ROWS, m0 = blockIdx.y * MT;
  const int len = f32_part_length(K), slabs = (len + FR_SLAB - 1) / FR_SLAB;

  auto load_w = [&](int slab, int stage) {
    float* dst = smem + stage * Rows::STAGE;
    // 16 parts x ROWS rows x 8 words of 16 bytes; eight neighbouring threads copy 128 bytes of a row
#pragma unroll
    for (int i = 0; i < FP_PARTS * ROWS * (FR_SLAB / 4) / FR_THREADS; ++i) {
      const int c = i * FR_THREADS + tid;
      const int word = c & 7, r = (c >> 3) % ROWS, p = (c >> 3) / ROWS;
      const int in_part = slab * FR_SLAB + word * 4, k = p * len + in_part;
      const bool ok = in_part < len && k < K && n0 + r < N;
      f32_copy16(dst + (p * ROWS + r) * FR_STRIDE + word * 4, w + (ok ? (size_t)(n0 + r) * K + k : 0), ok);
    }
  };
  auto load_x = [&](int slab, int stage) {
    float* dst = smem + stage * Rows::STAGE + FP_PARTS * ROWS * FR_STRIDE;
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const int word = tid & 7, p = tid >> 3;
      const int in_part = slab * FR_SLAB + word * 4, k = p * len + in_part;
      const bool ok = in_part < len && k < K && m0 + m < M;
      f32_copy16(dst + (m * FP_PARTS + p) * FR_SLAB + word * 4, x + (ok ? (size_t)(m0 + m) * K + k : 0), ok);
    }
  };

  // Weights do not depend on the kernels before this one: as many slabs as the ring takes are asked for before the wait.
  const int first = slabs < FR_STAGES - 1 ? slabs : FR_STAGES - 1;
  for (int s = 0; s < first; ++s) load_w(s, s);
  pdl_wait();
  for (int s = 0; s < FR_STAGES - 1; ++s) {
    if (s < first) load_x(s, s);
    f32_commit();          // the first of these groups also holds the weights of all of them
  }

  float acc[R][MT];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int m = 0; m < MT; ++m) acc[r][m] = 0.f;
  for (int s = 0; s < slabs; ++s) {
    f32_wait<FR_STAGES - 2>();
    __syncthreads();       // slab s has arrived for everyone, and slab s - 1 has been read by everyone
    const int ahead = s + FR_STAGES - 1;
    if (ahead < slabs) {
      load_w(ahead, ahead % FR_STAGES);
      load_x(ahead, ahead % FR_STAGES);
    }
    f32_commit();
    const float* stage = smem + (s % FR_STAGES) * Rows::STAGE;
    const float* ws = stage + (part * ROWS + row) * FR_STRIDE;
    const float* xs = stage + FP_PARTS * ROWS * FR_STRIDE + part * FR_SLAB;
    auto quad = [&](int i) {
      float4 b[R];
#pragma unroll
      for (int r = 0; r < R; ++r) b[r] = *reinterpret_cast<const float4*>(ws + r * 8 * FR_STRIDE + i);
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const float4 a = *reinterpret_cast<const float4*>(xs + m * FP_PARTS * FR_SLAB + i);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          acc[r][m] = fmaf(a.x, b[r].x, acc[r][m]);
          acc[r][m] = fmaf(a.y, b[r].y, acc[r][m]);
          acc[r][m] = fmaf(a.z, b[r].z, acc[r][m]);
          acc[r][m] = fmaf(a.w, b[r].w, acc[r][m]);
        }
      }
    };
    if constexpr (SHORT) {
      for (int i = 0; i < len; i += 4) quad(i);
    } else {
#pragma unroll
      for (int i = 0; i < FR_SLAB; i += 4) quad(i);
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const float p1 = __shfl_sync(0xffffffffu, acc[r][m], row + 8), p2 = __shfl_sync(0xffffffffu, acc[r][m], row + 16),
                  p3 = __shfl_sync(0xffffffffu, acc[r][m], row + 24);
      if (lane < 8) sums[tid >> 5][r * 8 + row][m] = ((acc[r][m] + p1) + p2) + p3;
    }
  __syncthreads();
  for (int o = tid; o < ROWS * MT; o += FR_THREADS) {
    const int r = o % ROWS, m = o / ROWS;
    if (n0 + r < N && m0 + m < M)
      out[(size_t)(m0 + m) * N + n0 + r] = ((sums[0][r][m] + sums[1][r][m]) + sums[2][r][m]) + sums[3][r][m];
  }
}

template <int MT, int R, bool SHORT>
static int launch_rows_form(const float* x, const float* w, float* out, int M, int N, int K, cudaStream_t stream) {
  using Rows = F32Rows<MT, R>;
  const int most = FR_STAGES * Rows::STAGE * (int)sizeof(float);
  static bool ready[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !ready[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(gemm_f32_rows_kernel<MT, R, SHORT>, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    if (e != cudaSuccess) return (int)e;
    if (dev < 64) ready[dev] = true;
  }
  // fewer slabs than stages: room for those alone, so that more CTAs fit an SM
  const int slabs = (f32_part_length(K) + FR_SLAB - 1) / FR_SLAB, smem = slabs < FR_STAGES ? most / FR_STAGES * slabs : most;
  const dim3 grid((N + Rows::ROWS - 1) / Rows::ROWS, (M + MT - 1) / MT);
  return launch(gemm_f32_rows_kernel<MT, R, SHORT>, grid, FR_THREADS, smem, stream, x, w, out, M, N, K);
}

template <int MT, int R>
static int launch_rows(const float* x, const float* w, float* out, int M, int N, int K, cudaStream_t stream) {
  return f32_part_length(K) < FR_SLAB ? launch_rows_form<MT, R, true>(x, w, out, M, N, K, stream)
                                      : launch_rows_form<MT, R, false>(x, w, out, M, N, K, stream);
}

// -------------------------------------------------------------------------------------------------- more rows
constexpr int FT_M = 32, FT_N = 64, FT_OWN = 4, FT_K = 32, FT_STRIDE = FT_K + 4, FT_STAGES = 3;
constexpr int FT_THREADS = (FT_M / FT_OWN) * (FT_N / FT_OWN), FT_STAGE = (FT_M + FT_N) * FT_STRIDE;     // floats

// WHOLE: parts are whole steps of 32 k; else a step may hold the ends of several.
template <int SPLIT, bool WHOLE>
__global__ void __launch_bounds__(FT_THREADS, 4) gemm_f32_tile_kernel(const float* x, const float* __restrict__ w, float* out,
                                                                   int M, int N, int K) {
  static_assert(SPLIT == 1 || SPLIT == 4, "all groups of K in one CTA, or one in each");
  constexpr int BM = FT_M, BN = FT_N, TM = FT_OWN, TN = FT_OWN;
  constexpr int THREADS = FT_THREADS, GROUPS = 4 / SPLIT, OUTS = TM * TN;
  extern __shared__ float smem[];
  float* kept = smem + FT_STAGES * FT_STAGE;           // SPLIT 4: [output of a thread][thread]
  pdl_trigger();
  const int tid = threadIdx.x;
  const int tx = tid % (BN / TN), ty = tid / (BN / TN);
  const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM;
  const int len = f32_part_length(K), range = GROUPS * 4 * len;           // k of a part, and of this CTA
  const int k_first = blockIdx.z * range, mine = max(0, min(range, K - k_first)), total = (mine + FT_K - 1) / FT_K;

  // Steps of 32 k, whatever parts they hold; either side (x or w) keeps its place, because the first steps of w are asked
  // for before x may be read. Zeros beyond the CTA's range and the matrix; parts beyond the matrix would add nothing
  // and are left out.
  constexpr int WORDS = FT_K / 4;
  auto load = [&](int& at, int rows, int r0, int limit, const float* src, float* dst) {
#pragma unroll
    for (int c = tid; c < rows * WORDS; c += THREADS) {
      const int word = c % WORDS, r = c / WORDS, k = k_first + at + word * 4;
      const bool ok = at + word * 4 < mine && r0 + r < limit;
      f32_copy16(dst + r * FT_STRIDE + word * 4, src + (ok ? (size_t)(r0 + r) * K + k : 0), ok);
    }
    at += FT_K;
  };
  int of_x = 0, of_w = 0;
  auto load_x = [&](int stage) { load(of_x, BM, m0, M, x, smem + stage * FT_STAGE); };
  auto load_w = [&](int stage) { load(of_w, BN, n0, N, w, smem + stage * FT_STAGE + BM * FT_STRIDE); };
#pragma unroll
  for (int s = 0; s < FT_STAGES - 1; ++s) load_w(s);        // weights first
  pdl_wait();
#pragma unroll
  for (int s = 0; s < FT_STAGES - 1; ++s) { load_x(s); f32_commit(); }

  float acc[TM][TN], group[TM][TN], sum[TM][TN];        // of a part, of a group, of the groups so far
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = group[i][j] = sum[i][j] = 0.f;
  auto end_part = [&]() {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) { group[i][j] += acc[i][j]; acc[i][j] = 0.f; }
  };
  auto end_group = [&]() {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) { sum[i][j] += group[i][j]; group[i][j] = 0.f; }
  };
  int stage = 0, part = 0, left = len / 4, ahead = (mine + 3) / 4;       // of the part and of all, in steps of four
  for (int step = 0; step < total; ++step) {
    f32_wait<FT_STAGES - 2>();
    __syncthreads();
    if (step + FT_STAGES - 1 < total) {
      const int free = stage == 0 ? FT_STAGES - 1 : stage - 1;      // read in the step before this one
      load_x(free);
      load_w(free);
    }
    f32_commit();
    const float* as = smem + stage * FT_STAGE + ty * FT_STRIDE;
    const float* bs = smem + stage * FT_STAGE + (BM + tx) * FT_STRIDE;
    stage = stage == FT_STAGES - 1 ? 0 : stage + 1;
    auto four = [&](int k) {
      float4 a[TM];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(as + i * (BM / TM) * FT_STRIDE + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const float4 v = *reinterpret_cast<const float4*>(bs + j * (BN / TN) * FT_STRIDE + k);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].x, v.x, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].y, v.y, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].z, v.z, acc[i][j]);
#pragma unroll
        for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].w, v.w, acc[i][j]);
      }
    };
    auto forward = [&](int fours_done) {
      left -= fours_done;
      if (left == 0) {
        left = len / 4;
        end_part();
        if ((++part & 3) == 0) end_group();
      }
    };
    if constexpr (WHOLE) {
#pragma unroll
      for (int q = 0; q < WORDS; ++q) four(4 * q);
      forward(WORDS);
    } else {
      const int fours = ahead < WORDS ? ahead : WORDS;
      ahead -= fours;
      for (int done = 0; done < fours;) {
        const int run = left < fours - done ? left : fours - done;
        if (run == WORDS) {
#pragma unroll
          for (int q = 0; q < WORDS; ++q) four(4 * q);
        } else {
          for (int q = 0; q < run; ++q) four(4 * (done + q));
        }
        done += run;
        forward(run);
      }
    }
  }
  end_part();         // (of a part that the matrix ends in; else they add zeros)
  end_group();
  f32_wait<0>();
  auto store = [&](int o, float v) {
    const int r = m0 + ty + (o / TN) * (BM / TM), c = n0 + tx + (o % TN) * (BN / TN);
    if (r < M && c < N) out[(size_t)r * N + c] = v;
  };
  if (SPLIT == 1) {
#pragma unroll
    for (int o = 0; o < OUTS; ++o) store(o, sum[o / TN][o % TN]);
  } else {
#pragma unroll
    for (int o = 0; o < OUTS; ++o) kept[o * THREADS + tid] = sum[o / TN][o % TN];
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    const float* of_group[4];
#pragma unroll
    for (int g = 0; g < 4; ++g) of_group[g] = cluster.map_shared_rank(kept, g) + tid;
    constexpr int SHARE = OUTS / SPLIT;
#pragma unroll 4
    for (int o = (int)blockIdx.z * SHARE; o < ((int)blockIdx.z + 1) * SHARE; ++o)
      store(o, ((of_group[0][o * THREADS] + of_group[1][o * THREADS]) + of_group[2][o * THREADS]) + of_group[3][o * THREADS]);
    cluster.sync();        // nobody leaves while its sums are still read
  }
}

template <int SPLIT, bool WHOLE>
static int launch_tile_form(const float* x, const float* w, float* out, int M, int N, int K, cudaStream_t stream) {
  auto kernel = gemm_f32_tile_kernel<SPLIT, WHOLE>;
  constexpr int own = (FT_STAGES * FT_STAGE + (SPLIT == 1 ? 0 : FT_M * FT_N)) * (int)sizeof(float);      // the ring, and the CTA's sums
  constexpr int sm_bytes = 228 * 1024;
  static bool ready[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !ready[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sm_bytes / 2 + 1024);
    if (e != cudaSuccess) return (int)e;
    if (dev < 64) ready[dev] = true;
  }
  if ((M + FT_M - 1) / FT_M > 65535) return TS_ERR_BAD_ARGUMENT;
  const dim3 grid((N + FT_N - 1) / FT_N, (M + FT_M - 1) / FT_M, SPLIT);
  // A grid of a few CTAs an SM starts while the kernel before it drains and piles up on the SMs that drain first: 64 rows of
  // 1,024 x 3,072, 128 CTAs, took 41 us on half of the SMs and take 24 us when no SM has room for two. So a CTA asks for as
  // much shared memory as lets no SM hold more than its share.
  const long long per_sm = ((long long)grid.x * grid.y * grid.z + 147) / 148;
  const int share = per_sm <= 3 ? sm_bytes / ((int)per_sm + 1) + 1024 : 0;
  const int smem = share > own ? share : own;
  if (SPLIT == 1) return launch(kernel, grid, FT_THREADS, smem, stream, x, w, out, M, N, K);
  return launch_cluster(kernel, grid, FT_THREADS, smem, stream, dim3(1, 1, SPLIT), x, w, out, M, N, K);
}

template <int SPLIT>
static int launch_tile(const float* x, const float* w, float* out, int M, int N, int K, cudaStream_t stream) {
  return f32_part_length(K) % FT_K == 0 ? launch_tile_form<SPLIT, true>(x, w, out, M, N, K, stream)
                                        : launch_tile_form<SPLIT, false>(x, w, out, M, N, K, stream);
}

}  // namespace ts

using namespace ts;

// `form`: 0 = chosen here; 1, 2 = a few rows, one or two weight rows a thread; 3, 4 = tiles, K over 1, 4 CTAs.
extern "C" int ts_gemm_f32(const float* x, const float* w, float* out, int M, int N, int K, int form, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || form < 0 || form > 4) return TS_ERR_BAD_ARGUMENT;
  if (K % 4 != 0 || (((uintptr_t)x | (uintptr_t)w) & 15) != 0) return TS_ERR_UNSUPPORTED;
  if (form == 0) {
    const long long tiles = (long long)((M + FT_M - 1) / FT_M) * ((N + FT_N - 1) / FT_N);
    // (K over 4 CTAs / over one: 128 rows of 4,096 x 1,024, 256 tiles, 39 / 42 us; 190 rows, 384 tiles, 53 / 53; 190 of
    // 6,144 x 1,024, 576 tiles, 79 / 67; 64 of 1,024 x 3,072, 32 tiles, 24 / 73. The cluster's meeting weighs more the
    // shorter K: 300 rows of 1,024 x 128, 160 tiles, 9.3 / 8.9; of 2,048 x 256, 320 tiles, 20 / 18; 40 of 4,096 x 64, 128
    // tiles, 6.7 / 5.4; 128 of 2,048 x 256, 128 tiles, 9.4 / 10.6)
    if (M <= 16) form = M > 2 && N >= 2048 ? 2 : 1;
    else form = tiles <= 400 && tiles <= 100 + K / 2 ? 4 : 3;
  }
  if (form <= 2) {
    if ((M + 7) / 8 > 65535) return TS_ERR_BAD_ARGUMENT;
    if (form == 1) {
      if (M == 1) return launch_rows<1, 1>(x, w, out, M, N, K, stream);
      if (M == 2) return launch_rows<2, 1>(x, w, out, M, N, K, stream);
      if (M <= 4) return launch_rows<4, 1>(x, w, out, M, N, K, stream);
      return launch_rows<8, 1>(x, w, out, M, N, K, stream);
    }
    return M <= 4 ? launch_rows<4, 2>(x, w, out, M, N, K, stream) : launch_rows<8, 2>(x, w, out, M, N, K, stream);
  }
  return form == 3 ? launch_tile<1>(x, w, out, M, N, K, stream) : launch_tile<4>(x, w, out, M, N, K, stream);
}
