// out[M, N] = x[M, K] * w[N, K]^T for a few rows and a large matrix, bf16, on the 5th-generation tensor cores with the
// operands' places changed: 128 rows of w are the A operand, 16 rows of x (zeros beyond M) the B operand, so that a tile of
// the accumulator is 128 columns of the output and no work is done for rows that are not there beyond the next 16 (more than
// 16 rows are several tiles, each of which reads w again; the library is faster there). Optionally the SwiGLU product of a
// merged matrix (64 gate and the 64 matching up rows make a tile).
//
// Bound by the stream of the weights. A CTA takes one tile of w and a slice of K; TMA copies of 128 rows x 64 k (16 KB,
// 128-byte swizzle) go through a ring of 5 stages, the first ones asked for before the wait for the kernels before
// this one; one thread issues the MMAs. No register holds a weight, so what is in flight does not depend on occupancy, and
// two CTAs fit an SM. The slices of a tile are a thread-block cluster: each CTA leaves its sums in shared memory (where
// the ring was) and the cluster adds them up in the order of the slices through distributed shared memory, so there is no
// scratch in global memory, no counter, and launches may overlap.
#define TS_PDL_CLASS PDL_SKINNY
#include <cooperative_groups.h>

#include "cache_map.cuh"
#include "tcgen05.cuh"
#include "launch_list.cuh"

namespace ts {
namespace cg = cooperative_groups;

constexpr int GR_BN = 128, GR_BK = 64, GR_XN = 16, GR_THREADS = 128, GR_MAX_SLICES = 8, GR_STAGES = 5;
constexpr uint32_t GR_W_BYTES = GR_BN * GR_BK * 2, GR_STAGE = GR_W_BYTES + GR_XN * GR_BK * 2;
constexpr uint32_t GR_TMEM_COLS = 32;       // the least there is; 16 are used
constexpr size_t GR_SMEM = GR_STAGES * (size_t)GR_STAGE + 1024;
static_assert(GR_SMEM >= TMEM_WAITING_SMEM, "beside no other kernel's CTA with tensor memory");
static_assert(GR_BN * GR_XN * 4 <= GR_STAGES * (int)GR_STAGE, "the sums take the place of the ring");

template <bool SWIGLU>
__global__ void __launch_bounds__(GR_THREADS) gemm_rows_tcgen05_kernel(const __grid_constant__ CUtensorMap map_x,
                                                                       const __grid_constant__ CUtensorMap map_w,
                                                                       bf16* __restrict__ out, int all_rows, int N, int K,
                                                                       int* __restrict__ error_flag) {
  constexpr int STAGES = GR_STAGES, XN = GR_XN, OUT = SWIGLU ? GR_BN / 2 : GR_BN;
  // instruction descriptor: D = f32, A = B = bf16, both K-major, N = XN, M = 128
  constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(XN >> 3) << 17) | ((uint32_t)(GR_BN >> 4) << 24);
  extern __shared__ unsigned char smem_raw[];
  unsigned char* ring = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full_bar[STAGES];
  __shared__ __align__(8) uint64_t empty_bar[STAGES];
  __shared__ __align__(8) uint64_t acc_full;
  __shared__ uint32_t tmem_base_slot;
  __shared__ int failed;

  pdl_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slices = gridDim.y, slice = blockIdx.y, n0 = blockIdx.x * OUT;
  const int m0 = blockIdx.z * XN, M = min(XN, all_rows - m0);       // this tile's rows
  out += (size_t)m0 * N;
  const int all_kb = (K + GR_BK - 1) / GR_BK;
  const int kb0 = (int)((long long)all_kb * slice / slices), num_kb = (int)((long long)all_kb * (slice + 1) / slices) - kb0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    mbar_init(&acc_full, 1);
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(&tmem_base_slot, GR_TMEM_COLS);      // in front of the wait: see TMEM_WAITING_SMEM
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_slot;

  if (warp == 0) {
    // ---------------- TMA producer (one lane)
    if (lane == 0 && !wait_test_unarmed()) {
      auto load_w = [&](int i) {
        const int s = i % STAGES;
        unsigned char* a = ring + (size_t)s * GR_STAGE;
        mbar_expect_tx(&full_bar[s], GR_STAGE);
        tma_load_2d(a, &map_w, &full_bar[s], (kb0 + i) * GR_BK, n0);
        if constexpr (SWIGLU) tma_load_2d(a + GR_W_BYTES / 2, &map_w, &full_bar[s], (kb0 + i) * GR_BK, N + n0);      // boxes of 64 rows
      };
      const int early = num_kb < STAGES ? num_kb : STAGES;
      for (int i = 0; i < early; ++i) load_w(i);
      pdl_wait();
      int i = 0;
      for (; i < num_kb; ++i) {
        const int s = i % STAGES;
        if (i >= early) {
          if (!mbar_wait(&empty_bar[s], ((i / STAGES) & 1) ^ 1)) { *(volatile int*)&failed = 1; break; }
          load_w(i);
        }
        tma_load_2d(ring + (size_t)s * GR_STAGE + GR_W_BYTES, &map_x, &full_bar[s], (kb0 + i) * GR_BK, m0);
      }
      // after a failure: copies in flight may still land in this CTA's shared memory
      if (*(volatile int*)&failed)
        for (int j = i > STAGES ? i - STAGES : 0; j < i; ++j) mbar_wait(&full_bar[j % STAGES], (j / STAGES) & 1);
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------- MMA issuer (one lane)
    if (lane == 0) {
      bool ok = true;
      for (int i = 0; i < num_kb && ok; ++i) {
        const int s = i % STAGES;
        ok = mbar_wait(&full_bar[s], (i / STAGES) & 1);
        if (!ok) { *(volatile int*)&failed = 1; break; }
        tc_fence_after();
        const uint32_t a_addr = smem_u32(ring + (size_t)s * GR_STAGE);
        const uint64_t adesc = sw128_desc(a_addr), bdesc = sw128_desc(a_addr + GR_W_BYTES);
#pragma unroll
        for (int k = 0; k < GR_BK / 16; ++k) umma_bf16(tmem, adesc + 2 * k, bdesc + 2 * k, IDESC, (i | k) != 0);
        umma_commit(&empty_bar[s]);
      }
      if (ok) umma_commit(&acc_full);
    }
    __syncwarp();
  }

  // ---------------- epilogue, all warps: thread = row of the tile = column of the output (SWIGLU: gate or up of one)
  pdl_wait();
  if (!mbar_wait(&acc_full, 0)) {
    if (lane == 0) atomicExch(error_flag, WAIT_FAILED_GEMM_TCGEN05);
  }
  tc_fence_after();
  __syncthreads();         // the ring is free: all its copies have arrived and all MMAs have read them
  float* sums = reinterpret_cast<float*>(ring);        // [row of x][row of the tile]
  {
    uint32_t v[32];
    tmem_ld_32(tmem + ((uint32_t)(warp * 32) << 16), v);
#pragma unroll
    for (int m = 0; m < XN; ++m) {
      if (m < M) {
        if (!SWIGLU && slices == 1) {
          if (n0 + (int)threadIdx.x < N) out[(size_t)m * N + n0 + threadIdx.x] = from_float<bf16>(__uint_as_float(v[m]));
        } else {
          sums[m * GR_BN + threadIdx.x] = __uint_as_float(v[m]);
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, GR_TMEM_COLS);
  if (!SWIGLU && slices == 1) return;
  cg::cluster_group cluster = cg::this_cluster();
  if (slices > 1) cluster.sync();
  const float* of_slice[GR_MAX_SLICES];
#pragma unroll
  for (int q = 0; q < GR_MAX_SLICES; ++q) of_slice[q] = slices > 1 && q < slices ? cluster.map_shared_rank(sums, q) : sums;
  // four neighbouring columns a thread: a trip to another CTA's shared memory costs the same for one word or for four
  constexpr int QUADS = OUT / 4;
#pragma unroll 2
  for (int idx = slice * GR_THREADS + threadIdx.x; idx < QUADS * M; idx += slices * GR_THREADS) {
    const int m = idx / QUADS, row = idx % QUADS * 4;
    float4 v[GR_MAX_SLICES], u[SWIGLU ? GR_MAX_SLICES : 1];
#pragma unroll
    for (int q = 0; q < GR_MAX_SLICES; ++q)
      if (q < slices) {
        v[q] = *reinterpret_cast<const float4*>(of_slice[q] + m * GR_BN + row);
        if constexpr (SWIGLU) u[q] = *reinterpret_cast<const float4*>(of_slice[q] + m * GR_BN + OUT + row);
      }
    float s[4] = {0.f, 0.f, 0.f, 0.f}, up[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int q = 0; q < GR_MAX_SLICES; ++q)
      if (q < slices) {        // the order of the slices
        s[0] += v[q].x; s[1] += v[q].y; s[2] += v[q].z; s[3] += v[q].w;
        if constexpr (SWIGLU) { up[0] += u[q].x; up[1] += u[q].y; up[2] += u[q].z; up[3] += u[q].w; }
      }
    if constexpr (SWIGLU) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        // rounding points of the separate kernels: product -> bf16, silu -> bf16, times up -> bf16
        const float gv = round_to<bf16>(s[e]), uv = round_to<bf16>(up[e]);
        s[e] = round_to<bf16>(gv / (1.f + expf(-gv))) * uv;
      }
    }
    bf16* o = out + (size_t)m * N + n0 + row;
    if (N % 4 == 0 && n0 + row < N) {
      Quad<bf16>::store(o, s);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (n0 + row + e < N) o[e] = from_float<bf16>(s[e]);
    }
  }
  if (slices > 1) cluster.sync();      // nobody leaves while its sums are still read
}

// rows x K bf16 row-major; boxes of box_rows x 64, 128-byte swizzle, zero fill outside.
static bool rows_map(CUtensorMap* map, const void* base, int rows, int K, int box_rows, CUtensorMapL2promotion promotion) {
  DtEncodeFn fn = dt_encode_fn();
  if (fn == nullptr) return false;
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)K * 2};
  cuuint32_t box[2] = {(cuuint32_t)GR_BK, (cuuint32_t)box_rows};
  cuuint32_t elem[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, promotion, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <bool SWIGLU>
static int launch_rows_tc(const void* x, const void* w, bf16* out, int M, int N, int K, int slices, int* error_flag, cudaStream_t stream) {
  constexpr int OUT = SWIGLU ? GR_BN / 2 : GR_BN;
  CUtensorMap mx, mw;
  if (!rows_map(&mx, x, M, K, GR_XN, CU_TENSOR_MAP_L2_PROMOTION_L2_128B) ||
      !rows_map(&mw, w, SWIGLU ? 2 * N : N, K, OUT, CU_TENSOR_MAP_L2_PROMOTION_L2_256B))
    return TS_ERR_UNSUPPORTED;
  auto kern = gemm_rows_tcgen05_kernel<SWIGLU>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GR_SMEM);
  if (e != cudaSuccess) return (int)e;
  const dim3 grid((N + OUT - 1) / OUT, slices, (M + GR_XN - 1) / GR_XN);
  if (slices == 1) return launch(kern, grid, GR_THREADS, GR_SMEM, stream, mx, mw, out, M, N, K, error_flag);
  return launch_cluster(kern, grid, GR_THREADS, GR_SMEM, stream, dim3(1, slices), mx, mw, out, M, N, K, error_flag);
}

}  // namespace ts

using namespace ts;

// M <= 64, K % 8 == 0, any N; slices of K: 1 to 8 (at least one block of 64 each). swiglu: w is [2 N, K] (gate rows, then
// up rows) and out = silu(gate) * up, [M, N].
extern "C" int ts_gemm_rows_tcgen05(const void* x, const void* w, void* out, int M, int N, int K, int swiglu, int slices,
                                    int* error_flag, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (slices < 1 || slices > GR_MAX_SLICES) return TS_ERR_BAD_ARGUMENT;
  if (M > 64 || K <= 0 || K % 8 != 0 || slices > (K + GR_BK - 1) / GR_BK || error_flag == nullptr) return TS_ERR_UNSUPPORTED;
  if (((uintptr_t)x | (uintptr_t)w | (uintptr_t)out) & 15) return TS_ERR_UNSUPPORTED;        // copies of 16 bytes, stores of 8
  return swiglu ? launch_rows_tc<true>(x, w, (bf16*)out, M, N, K, slices, error_flag, stream)
                : launch_rows_tc<false>(x, w, (bf16*)out, M, N, K, slices, error_flag, stream);
}
TS_LIST_ENTRY(ts_gemm_rows_tcgen05);
