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
// More rows: bound by the multiply-adds and, below some hundred rows, by the latency of the chains. A warp owns a tile of
// 32 x 64 outputs, 8 x 8 a thread (a thread reads 16 words of shared memory for 64 multiply-adds; the 4 x 4 tiles that this
// replaces read 32 for as many), and one stretch of K, so a CTA's four warps share a tile of outputs and nothing else: each
// copies its own rows of x and w, in steps of 16 k and three cp.async stages, and none waits for another before the sums
// meet in shared memory. Where the tiles are too few for the machine, a CTA takes one of the four groups, a warp one of its
// parts, and the groups' CTAs are a cluster that adds up through distributed shared memory; else a warp takes a group and
// keeps its parts' sums in shared memory. Parts shorter than a step (K up to 192), and many tiles whose parts are no whole steps
// (ts_gemm_f32), go to a kernel of thread tiles of 4 x 4
// whose steps hold several parts (600 rows of 10,000 x 100 50 us, in steps of their own 73). Measured, 4 x 4 tiles for all / now: 64 rows of
// 1,024 x 2,048 15.1 / 12.3 us, of 1,024 x 3,072 21.1 / 16.7, 128 rows of 4,096 x 1,024 39.9 / 32.7, of 1,024 x 3,072 32.8 / 24.6,
// 190 rows of 6,144 x 1,024 70.8 / 64.5, 600 rows 216 / 203 (37 TFLOP/s: two or three warps a scheduler, which issue 72 % of
// the time, 78 % of it multiply-adds; two at a time, fma.rn.f32x2, come to no more than 45 TFLOP/s in registers alone, one
// at a time to 66). K over 4 CTAs / over one: 64 rows of 4,096 x 1,024, 128 tiles, 21 / 21 us, of 6,144 x 1,024, 192 tiles, 31 / 32;
// 128 rows, 256 and 384 tiles, 41 / 33 and 58 / 52; 600 rows of 1,024 x 2,048, 304 tiles, 76 / 93; 64 and 128 rows of 2,048 x
// 256, 64 and 128 tiles, 5.9 / 7.6 and 12.3 / 7.8: the cluster's meeting weighs more the shorter K.
#define TS_PDL_CLASS PDL_OTHER
#include <cooperative_groups.h>

#include <type_traits>

#include "common.cuh"
#include "launch_list.cuh"

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
constexpr int FT_M = 32, FT_N = 64, FT_OWN = 8, FT_K = 16, FT_TEAMS = 4, FT_STAGES = 3;
constexpr int FT_THREADS = FT_TEAMS * 32, FT_STAGE = (FT_M + FT_N) * FT_K;       // floats of a warp's stage
constexpr int FT_SUM_STRIDE = FT_N + 8, FT_SUMS = FT_M * FT_SUM_STRIDE;          // of a warp's sums: no two lanes in one bank
static_assert(FT_SUMS <= FT_STAGES * FT_STAGE, "with K over a cluster the sums take the place of the ring");

// A warp's tile in one stage: rows of 16 k in four words of 16 bytes, whose places within a row are swapped by the row, so
// that eight neighbouring rows read at the same word lie in different banks.
__device__ __forceinline__ int f32_word_at(int row, int word) { return row * FT_K + ((word ^ ((row >> 1) & 3)) << 2); }

// SPLIT 1: warp = one of the four groups of K. SPLIT 4: the CTA has one group, warp = one of its parts.
// CTAS: CTAs of an SM, what the registers of a thread are held to.
template <int SPLIT, int CTAS>
__global__ void __launch_bounds__(FT_THREADS, CTAS) gemm_f32_tile_kernel(const float* x, const float* __restrict__ w,
                                                                                     float* out, int M, int N, int K) {
  static_assert(SPLIT == 1 || SPLIT == 4, "all groups of K in one CTA, or one in each");
  constexpr int PARTS = SPLIT == 1 ? 4 : 1, OWN = FT_OWN;       // parts a warp goes through
  extern __shared__ float smem[];
  pdl_trigger();
  const int lane = threadIdx.x & 31, team = threadIdx.x >> 5;
  const int tx = lane & 7, ty = lane >> 3;
  const int n0 = blockIdx.x * FT_N, m0 = blockIdx.y * FT_M;
  const int len = f32_part_length(K), first_part = SPLIT == 1 ? 4 * team : 4 * blockIdx.z + team;
  float* ring = smem + team * (FT_STAGES * FT_STAGE);
  float* sums = SPLIT == 1 ? smem + FT_TEAMS * (FT_STAGES * FT_STAGE) : smem;       // [team][row][column]

  // ---- copies: four lanes a row. A step holds 16 k of one part (fewer at its end); x and w keep their own places in the
  // sequence of steps, because the first steps of w are asked for before x may be read.
  const int row = lane >> 2, word = lane & 3;
  const float* x_row = x + (size_t)(m0 + row) * K + word * 4;
  const float* w_row = w + (size_t)(n0 + row) * K + word * 4;
  struct Place { int part, at, stage; };       // the next step: of which part, from which of its k, into which stage
  auto k_end = [&](int part) { return max(0, min(len, K - (first_part + part) * len)); };
  auto skip_empty = [&](Place& p) { while (p.part < PARTS && p.at >= k_end(p.part)) { ++p.part; p.at = 0; } };
  auto copy = [&](Place& p, auto rows, const float* src, int limit, int offset) {
    if (p.part < PARTS) {
      const int k = (first_part + p.part) * len + p.at;
      const bool ok = p.at + word * 4 < k_end(p.part);
      float* dst = ring + p.stage * FT_STAGE + offset;
#pragma unroll
      for (int i = 0; i < decltype(rows)::value / 8; ++i) {
        const bool in = ok && row + 8 * i < limit;
        f32_copy16(dst + f32_word_at(row + 8 * i, word), in ? src + (size_t)(8 * i) * K + k : w, in);
      }
      p.at += FT_K;
      p.stage = p.stage == FT_STAGES - 1 ? 0 : p.stage + 1;
      skip_empty(p);
    }
  };
  Place of_x = {0, 0, 0}, of_w = {0, 0, 0}, now = {0, 0, 0};
  skip_empty(of_x);
  of_w = now = of_x;
  auto load_x = [&]() { copy(of_x, std::integral_constant<int, FT_M>(), x_row, M - m0, 0); };
  auto load_w = [&]() { copy(of_w, std::integral_constant<int, FT_N>(), w_row, N - n0, FT_M * FT_K); };
#pragma unroll
  for (int s = 0; s < FT_STAGES - 1; ++s) load_w();        // weights first
  pdl_wait();
#pragma unroll
  for (int s = 0; s < FT_STAGES - 1; ++s) { load_x(); f32_commit(); }

  float acc[OWN][OWN];
#pragma unroll
  for (int i = 0; i < OWN; ++i)
#pragma unroll
    for (int j = 0; j < OWN; ++j) acc[i][j] = 0.f;
  float* my_sums = sums + team * FT_SUMS + ty * FT_SUM_STRIDE + tx;
  for (int part = 0; part < PARTS; ++part) {
    const int end = k_end(part);
    for (int at = 0; at < end; at += FT_K) {
      f32_wait<FT_STAGES - 2>();
      __syncwarp();        // the step's words have arrived for every lane, and the step before it has been read by every lane
      const float* as = ring + now.stage * FT_STAGE + ty * FT_K;
      const float* bs = ring + now.stage * FT_STAGE + FT_M * FT_K + tx * FT_K;
      now.stage = now.stage == FT_STAGES - 1 ? 0 : now.stage + 1;
      load_x();
      load_w();
      f32_commit();
      auto four = [&](int q) {
        float4 a[OWN];
#pragma unroll
        for (int i = 0; i < OWN; ++i)       // rows ty + 4 i
          a[i] = *reinterpret_cast<const float4*>(as + 4 * i * FT_K + ((q ^ (((ty >> 1) + 2 * i) & 3)) << 2));
#pragma unroll
        for (int j = 0; j < OWN; ++j) {     // rows tx + 8 j
          const float4 b = *reinterpret_cast<const float4*>(bs + 8 * j * FT_K + ((q ^ ((tx >> 1) & 3)) << 2));
#pragma unroll
          for (int i = 0; i < OWN; ++i) acc[i][j] = fmaf(a[i].x, b.x, acc[i][j]);
#pragma unroll
          for (int i = 0; i < OWN; ++i) acc[i][j] = fmaf(a[i].y, b.y, acc[i][j]);
#pragma unroll
          for (int i = 0; i < OWN; ++i) acc[i][j] = fmaf(a[i].z, b.z, acc[i][j]);
#pragma unroll
          for (int i = 0; i < OWN; ++i) acc[i][j] = fmaf(a[i].w, b.w, acc[i][j]);
        }
      };
      if (end - at >= FT_K) {
#pragma unroll
        for (int q = 0; q < FT_K / 4; ++q) four(q);
      } else {
        for (int q = 0; q < (end - at) / 4; ++q) four(q);
      }
    }
    if (SPLIT == 1) {      // the part's sums join the group's, which wait in shared memory (nobody else touches these)
#pragma unroll
      for (int i = 0; i < OWN; ++i)
#pragma unroll
        for (int j = 0; j < OWN; ++j) {
          float* s = my_sums + 4 * i * FT_SUM_STRIDE + 8 * j;
          *s = part == 0 ? acc[i][j] : *s + acc[i][j];
          acc[i][j] = 0.f;
        }
    }
  }
  f32_wait<0>();
  if (SPLIT == 4) {
    __syncthreads();       // every warp has read its ring to the end
#pragma unroll
    for (int i = 0; i < OWN; ++i)
#pragma unroll
      for (int j = 0; j < OWN; ++j) my_sums[4 * i * FT_SUM_STRIDE + 8 * j] = acc[i][j];
  }
  __syncthreads();
  // ---- the four sums of an output (of groups, or of the group's parts) added left to right, four neighbouring columns a
  // thread
  auto add_up = [&](const float* const (&of)[4], int o) {
    float4 s = *reinterpret_cast<const float4*>(of[0] + o);
#pragma unroll
    for (int q = 1; q < 4; ++q) {
      const float4 v = *reinterpret_cast<const float4*>(of[q] + o);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    return s;
  };
  const bool by_fours = N % 4 == 0 && ((uintptr_t)out & 15) == 0;
  auto store = [&](int r, int c, float4 s) {
    if (m0 + r >= M) return;
    float* o = out + (size_t)(m0 + r) * N + n0 + c;
    if (by_fours && n0 + c < N) {
      *reinterpret_cast<float4*>(o) = s;
    } else {
      const float v[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (n0 + c + e < N) o[e] = v[e];
    }
  };
  constexpr int QUADS = FT_N / 4;
  const float* of_team[4] = {sums, sums + FT_SUMS, sums + 2 * FT_SUMS, sums + 3 * FT_SUMS};
  if (SPLIT == 1) {
    for (int q = threadIdx.x; q < FT_M * QUADS; q += FT_THREADS) {
      const int r = q / QUADS, c = q % QUADS * 4;
      store(r, c, add_up(of_team, r * FT_SUM_STRIDE + c));
    }
  } else {
    for (int q = threadIdx.x; q < FT_M * QUADS; q += FT_THREADS) {      // in place of the first part's
      const int o = q / QUADS * FT_SUM_STRIDE + q % QUADS * 4;
      *reinterpret_cast<float4*>(sums + o) = add_up(of_team, o);
    }
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    const float* of_group[4];
#pragma unroll
    for (int g = 0; g < 4; ++g) of_group[g] = cluster.map_shared_rank(sums, g);
    constexpr int SHARE = FT_M / SPLIT;        // rows
    for (int q = threadIdx.x; q < SHARE * QUADS; q += FT_THREADS) {
      const int r = (int)blockIdx.z * SHARE + q / QUADS, c = q % QUADS * 4;
      store(r, c, add_up(of_group, r * FT_SUM_STRIDE + c));
    }
    cluster.sync();        // nobody leaves while its sums are still read
  }
}

// ----------------------------------------------------------------------- more rows, parts that are no whole steps
constexpr int FS_OWN = 4, FS_K = 32, FS_STRIDE = FS_K + 4, FS_STAGES = 3;
constexpr int FS_THREADS = (FT_M / FS_OWN) * (FT_N / FS_OWN), FS_STAGE = (FT_M + FT_N) * FS_STRIDE;     // floats

// Thread tiles of 4 x 4 whose CTA goes through K in steps of 32 k that hold several parts each.
template <int SPLIT>
__global__ void __launch_bounds__(FS_THREADS, 4) gemm_f32_short_kernel(const float* x, const float* __restrict__ w, float* out, int M,
                                                                    int N, int K) {
  static_assert(SPLIT == 1 || SPLIT == 4, "all groups of K in one CTA, or one in each");
  constexpr int BM = FT_M, BN = FT_N, TM = FS_OWN, TN = FS_OWN;
  constexpr int THREADS = FS_THREADS, GROUPS = 4 / SPLIT, OUTS = TM * TN;
  extern __shared__ float smem[];
  float* kept = smem + FS_STAGES * FS_STAGE;           // SPLIT 4: [output of a thread][thread]
  pdl_trigger();
  const int tid = threadIdx.x;
  const int tx = tid % (BN / TN), ty = tid / (BN / TN);
  const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM;
  const int len = f32_part_length(K), range = GROUPS * 4 * len;           // k of a part, and of this CTA
  const int k_first = blockIdx.z * range, mine = max(0, min(range, K - k_first)), total = (mine + FS_K - 1) / FS_K;

  // Steps of 32 k, whatever parts they hold; either side (x or w) keeps its place, because the first steps of w are asked
  // for before x may be read. Zeros beyond the CTA's range and the matrix; parts beyond the matrix would add nothing
  // and are left out.
  constexpr int WORDS = FS_K / 4;
  auto load = [&](int& at, int rows, int r0, int limit, const float* src, float* dst) {
#pragma unroll
    for (int c = tid; c < rows * WORDS; c += THREADS) {
      const int word = c % WORDS, r = c / WORDS, k = k_first + at + word * 4;
      const bool ok = at + word * 4 < mine && r0 + r < limit;
      f32_copy16(dst + r * FS_STRIDE + word * 4, src + (ok ? (size_t)(r0 + r) * K + k : 0), ok);
    }
    at += FS_K;
  };
  int of_x = 0, of_w = 0;
  auto load_x = [&](int stage) { load(of_x, BM, m0, M, x, smem + stage * FS_STAGE); };
  auto load_w = [&](int stage) { load(of_w, BN, n0, N, w, smem + stage * FS_STAGE + BM * FS_STRIDE); };
#pragma unroll
  for (int s = 0; s < FS_STAGES - 1; ++s) load_w(s);        // weights first
  pdl_wait();
#pragma unroll
  for (int s = 0; s < FS_STAGES - 1; ++s) { load_x(s); f32_commit(); }

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
    f32_wait<FS_STAGES - 2>();
    __syncthreads();
    if (step + FS_STAGES - 1 < total) {
      const int free = stage == 0 ? FS_STAGES - 1 : stage - 1;      // read in the step before this one
      load_x(free);
      load_w(free);
    }
    f32_commit();
    const float* as = smem + stage * FS_STAGE + ty * FS_STRIDE;
    const float* bs = smem + stage * FS_STAGE + (BM + tx) * FS_STRIDE;
    stage = stage == FS_STAGES - 1 ? 0 : stage + 1;
    auto four = [&](int k) {
      float4 a[TM];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(as + i * (BM / TM) * FS_STRIDE + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const float4 v = *reinterpret_cast<const float4*>(bs + j * (BN / TN) * FS_STRIDE + k);
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

// A grid of a few CTAs an SM starts while the kernel before it drains and piles up on the SMs that drain first: 64 rows of
// 1,024 x 3,072, 128 CTAs, took 41 us on half of the SMs and take 24 us when no SM has room for two. So a CTA asks for as
// much shared memory as lets no SM hold more than its share.
constexpr int F32_SM_BYTES = 228 * 1024;
template <typename Kernel>
static int launch_spread(Kernel kernel, dim3 grid, int threads, int own, int cluster, const float* x, const float* w, float* out, int M,
                         int N, int K, cudaStream_t stream) {
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, F32_SM_BYTES / 2 + 1024);
  if (e != cudaSuccess) return (int)e;
  const long long per_sm = ((long long)grid.x * grid.y * grid.z + 147) / 148;
  const int share = per_sm <= 3 ? F32_SM_BYTES / ((int)per_sm + 1) + 1024 : 0;
  const int smem = share > own ? share : own;
  if (cluster == 1) return launch(kernel, grid, threads, smem, stream, x, w, out, M, N, K);
  return launch_cluster(kernel, grid, threads, smem, stream, dim3(1, 1, cluster), x, w, out, M, N, K);
}

// How many CTAs one SM runs of a grid of `ctas`, `per` of them at a time.
static long long f32_rounds(long long ctas, int per) { return (ctas + 148 * per - 1) / (148 * per) * per; }

template <int SPLIT>
static int launch_tile(bool fine, const float* x, const float* w, float* out, int M, int N, int K, cudaStream_t stream) {
  if ((M + FT_M - 1) / FT_M > 65535) return TS_ERR_BAD_ARGUMENT;
  const dim3 grid((N + FT_N - 1) / FT_N, (M + FT_M - 1) / FT_M, SPLIT);
  if (fine) {
    constexpr int own = (FS_STAGES * FS_STAGE + (SPLIT == 1 ? 0 : FT_M * FT_N)) * (int)sizeof(float);      // the ring, and the CTA's sums
    return launch_spread(gemm_f32_short_kernel<SPLIT>, grid, FS_THREADS, own, SPLIT, x, w, out, M, N, K, stream);
  }
  constexpr int own = FT_TEAMS * (FT_STAGES * FT_STAGE + (SPLIT == 1 ? FT_SUMS : 0)) * (int)sizeof(float);
  // Two CTAs an SM have registers to look further ahead, three hide more by taking turns; what counts more is the CTAs that an
  // SM is given in the end (see f32_rounds). K over four CTAs, 1,024 columns and K = 2,048, two / three: 128 rows (256
  // CTAs) 17.6 / 20.0 us, 190 rows (384) 33.7 / 27.1, 600 rows (1,216) 80.7 / 76.4; 64 rows of 4,096 x 1,024 (512) 21.3 / 26.4.
  const long long ctas = (long long)grid.x * grid.y * grid.z;
  if (SPLIT == 4 && f32_rounds(ctas, 3) <= f32_rounds(ctas, 2))
    return launch_spread(gemm_f32_tile_kernel<SPLIT, SPLIT == 4 ? 3 : 2>, grid, FT_THREADS, own, SPLIT, x, w, out, M, N, K, stream);
  return launch_spread(gemm_f32_tile_kernel<SPLIT, 2>, grid, FT_THREADS, own, SPLIT, x, w, out, M, N, K, stream);
}

}  // namespace ts

using namespace ts;

// `form`: 0 = chosen here; 1, 2 = a few rows, one or two weight rows a thread; 3, 4 = tiles of a warp, K over 1, 4 CTAs; 5, 6 =
// tiles of a CTA, likewise.
extern "C" int ts_gemm_f32(const float* x, const float* w, float* out, int M, int N, int K, int form, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || form < 0 || form > 6) return TS_ERR_BAD_ARGUMENT;
  if (K % 4 != 0 || (((uintptr_t)x | (uintptr_t)w) & 15) != 0) return TS_ERR_UNSUPPORTED;
  if (form == 0) {
    const long long tiles = (long long)((M + FT_M - 1) / FT_M) * ((N + FT_N - 1) / FT_N);
    // K over four CTAs where an SM is then given less than a quarter as many CTAs' worth, the cluster's meeting counted as 384 k
    // (192 of a short K); many tiles, or a few hundred of a short K, fill the machine as they are (640 tiles of K = 1,024 81 / 88
    // us with one / four; 96 of K = 320 11.2 / 8.8).
    const long long four = f32_rounds(4 * tiles, 2) < f32_rounds(4 * tiles, 3) ? f32_rounds(4 * tiles, 2) : f32_rounds(4 * tiles, 3);
    const int part = f32_part_length(K);
    const bool split = part < FT_K ? tiles <= 400 && tiles <= 100 + K / 2
                                   : tiles <= (K < 512 ? 110 : 320) && four + (K < 512 ? 192.0 : 384.0) / K < 4.0 * f32_rounds(tiles, 1);
    // A warp's own steps end with each part, so parts that are no whole steps, or of which K is short, leave steps half empty. With
    // more tiles than run at once a CTA's tiles then are ahead (a warp's / a CTA's: 1,000 rows of 4,096 x 196 72 / 57 us, x 288
    // 95 / 79, x 448 128 / 118, x 512, whole steps, 119 / 127; 190 rows of 4,096 x 1,040 76 / 67), and with a tile for nearly every SM they are with K over four
    // CTAs (256 rows of 1,000 x 320 11.2 / 10.4).
    const bool ragged = (part <= 68 && part % 8 == 4) || part == 24;
    if (M <= 16) form = M > 2 && N >= 2048 ? 2 : 1;
    else if (part < FT_K) form = split ? 6 : 5;
    else if (split) form = 4;
    else if (tiles > 256 && (ragged || K <= 256)) form = 5;
    else form = ragged && tiles > 110 && tiles <= 148 ? 6 : 3;
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
  const bool fine = form > 4 || f32_part_length(K) < FT_K;
  return form & 1 ? launch_tile<1>(fine, x, w, out, M, N, K, stream) : launch_tile<4>(fine, x, w, out, M, N, K, stream);
}
TS_LIST_ENTRY(ts_gemm_f32);
