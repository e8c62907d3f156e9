// Next-token selection on the device: greedy argmax, temperature sampling, nucleus (top-p).
//
// Meaning of the options follows upstream src/tinyserve/sampling.py:56-102: temperature 0 is
// the argmax of the raw 32-bit logits; otherwise the token is drawn from softmax(logits / T)
// by the exponential race argmax_i p_i / E_i with E_i ~ Exp(1); with top_p < 1 only tokens are
// eligible whose more likely tokens together hold less than top_p of the mass (the most likely
// token always is), without renormalising. Differences: the noise comes from a counter-based
// generator (Philox4x32-10) keyed by the request's seed and indexed by (how many tokens the
// request has drawn, token id), so a request's tokens do not depend on its batch-mates, on
// chunking or on recomputation; tokens of exactly equal probability are kept or dropped
// together by top-p; the race is run on logit / T - log E_i, which orders the same way.
//
// A row is cut into chunks, one CTA each; the CTA that arrives last picks the winner among the
// chunks' winners, which meet in one array per device: launches without top-p that may run at the
// same time (on two streams) would share it. A row with top-p needs sums over the whole row, again
// and again, for the search of its threshold: its chunks are the CTAs of a cluster (one to eight, by
// the vocabulary) that keep their weights in registers (20 a thread: 163,840 tokens; a larger
// vocabulary is read from L2 each time) and add up their sums, and pick the winner, through
// distributed shared memory. Bound by the passes over the weights and the barrier of each: seven thresholds a pass, a warp none
// of whose weights lie between the bounds left leaves its sums where they are, the search starts from a bound that the mean
// weight gives, and as soon as no more than 1,024 weights are left between the bounds, every CTA sorts these and sums them up
// itself. Normal logits, top-p 0.95 at deviation 3 and 0.99 at 8, passes to the end (11 of them) / now: 151,936 tokens, 1 row
// 46.8, 30.5 / 39.2, 22.7 us, 64 rows 226, 158 / 192, 105, 256 rows 823, 572 / 698, 392; 32,768 tokens, 1 row 43.3, 31.1 / 31.8, 17.7, 256
// rows 172, 129 / 130, 81; 1,000 tokens, 1 row 15.5, 13.9 / 11.6, 8.9. (One CTA a row and two-way passes took 1,023 us for a row of
// 151,936.) Beyond 163,840 tokens nothing is sorted: 200,000 tokens 72.5 / 72.7.
#define TS_PDL_CLASS PDL_SAMPLING
#include <cooperative_groups.h>

#include "common.cuh"

namespace ts {
namespace cg = cooperative_groups;

constexpr int SM_THREADS = 1024;
constexpr int SM_MAX_ROWS = 4096;
constexpr int SM_MAX_CHUNKS = 32;

struct Best {
  float v;
  int i;
};
// Winners of the chunks, and an arrival counter per row that the last CTA puts back to zero.
static __device__ Best g_chunk_best[SM_MAX_ROWS * SM_MAX_CHUNKS];
static __device__ unsigned int g_row_arrivals[SM_MAX_ROWS];

__device__ __forceinline__ Best better(Best a, Best b) {
  if (b.i < 0) return a;
  if (a.i < 0) return b;
  if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
  return a;
}
__device__ __forceinline__ Best block_best(Best x, Best* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    Best y;
    y.v = __shfl_xor_sync(0xffffffffu, x.v, o);
    y.i = __shfl_xor_sync(0xffffffffu, x.i, o);
    x = better(x, y);
  }
  __syncthreads();
  if (lane == 0) scratch[warp] = x;
  __syncthreads();
  Best t;
  t.v = 0.f; t.i = -1;
  if (lane < nwarps) t = scratch[lane];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    Best y;
    y.v = __shfl_xor_sync(0xffffffffu, t.v, o);
    y.i = __shfl_xor_sync(0xffffffffu, t.i, o);
    t = better(t, y);
  }
  return t;
}
__device__ __forceinline__ float block_max(float v, float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  float t = (lane < nwarps) ? scratch[lane] : -INFINITY;
  return warp_max(t);
}

__device__ __forceinline__ void philox4x32_10(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, uint32_t k0,
                                              uint32_t k1, uint32_t out[4]) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t hi0 = __umulhi(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
    const uint32_t hi1 = __umulhi(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
    const uint32_t n0 = hi1 ^ c1 ^ k0, n2 = hi0 ^ c3 ^ k1;
    c0 = n0; c1 = lo1; c2 = n2; c3 = lo0;
    k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
  }
  out[0] = c0; out[1] = c1; out[2] = c2; out[3] = c3;
}

// exp(logit / T - max) with each step rounded on its own, so that the nucleus threshold found by
// the search and the later eligibility test see bit-identical values (no fused multiply-add).
__device__ __forceinline__ float scaled(float logit, float inv_t) { return __fmul_rn(logit, inv_t); }
__device__ __forceinline__ float weight_of(float logit, float inv_t, float mx) {
  return expf(__fsub_rn(scaled(logit, inv_t), mx));
}

// -log(u) with u uniform in (0, 1) on a 24-bit grid: never 0, never infinite.
__device__ __forceinline__ float exp1_from_bits(uint32_t x) {
  const float u = ((float)(x >> 8) + 0.5f) * (1.0f / 16777216.0f);
  return -logf(u);
}

// Best candidate of tokens [begin, end) (begin a multiple of 4) for one row.
// threshold: tokens with exp(z - mx) below it are not eligible (0 = all are).
__device__ __forceinline__ Best scan_range(const float* __restrict__ l, int begin, int end, float temp,
                                           float mx, float threshold, uint32_t k0, uint32_t k1, uint32_t d0,
                                           uint32_t d1) {
  Best best;
  best.v = 0.f; best.i = -1;
  if (!(temp > 0.f)) {
    // greedy: a thread's indices only grow, so "strictly greater" keeps the first maximum.
    float bv = -INFINITY;
    int bi = -1;
    if ((((uintptr_t)l) & 15) == 0) {
      const float4* l4 = reinterpret_cast<const float4*>(l);
      for (int i4 = begin / 4 + threadIdx.x; i4 * 4 < end; i4 += blockDim.x) {
        const int i = i4 * 4;
        if (i + 4 <= end) {
          const float4 v = l4[i4];
          if (v.x > bv) { bv = v.x; bi = i; }
          if (v.y > bv) { bv = v.y; bi = i + 1; }
          if (v.z > bv) { bv = v.z; bi = i + 2; }
          if (v.w > bv) { bv = v.w; bi = i + 3; }
        } else {
          for (int e = i; e < end; ++e)
            if (l[e] > bv) { bv = l[e]; bi = e; }
        }
      }
    } else {
      for (int i = begin + threadIdx.x; i < end; i += blockDim.x)
        if (l[i] > bv) { bv = l[i]; bi = i; }
    }
    if (bi < 0 && begin + (int)threadIdx.x < end) { bv = l[begin + threadIdx.x]; bi = begin + threadIdx.x; }  // all -inf / NaN
    best.v = bv; best.i = bi;
    return best;
  }
  const float inv_t = 1.f / temp;
  for (int i4 = begin / 4 + threadIdx.x; i4 * 4 < end; i4 += blockDim.x) {
    float z[4];
    bool eligible[4], any = false;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = i4 * 4 + e;
      z[e] = i < end ? scaled(l[i], inv_t) : 0.f;
      eligible[e] = i < end && (threshold <= 0.f || weight_of(l[i], inv_t, mx) >= threshold);
      any = any || eligible[e];
    }
    if (!any) continue;      // few tokens of a nucleus: no noise for the others
    uint32_t r[4];
    philox4x32_10((uint32_t)i4, d0, d1, 0u, k0, k1, r);
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (eligible[e]) {
        Best c; c.v = z[e] - logf(exp1_from_bits(r[e])); c.i = i4 * 4 + e;
        best = better(best, c);
      }
  }
  return best;
}

// The nucleus threshold of one row by the cluster of its CTAS chunks: the smallest bit pattern b in
// [0, bits(1.0)] with mass{weight > float(b)} < top_p * mass{all}. Tokens of [begin, end) are this CTA's.
constexpr int NUCLEUS_WAYS = 8, NUCLEUS_HELD = 20, NUCLEUS_HELD_SMALL = 4;
constexpr int NUCLEUS_LIST = SM_THREADS;      // weights that are sorted at the end, one a thread

struct NucleusShared {
  float scratch[33];
  float by_warp[NUCLEUS_WAYS - 1][32];
  float mine[2][NUCLEUS_WAYS];          // this CTA's sums (the last: how many weights lie between the bounds), read by the whole
                                        // cluster; alternating
  float whole[2][NUCLEUS_WAYS];         // the cluster's
  int listed[2];                        // this CTA's weights between the bounds, alternating ...
  float list[NUCLEUS_LIST];             // ... and the weights, in any order, if there are no more than these
  float sorted[NUCLEUS_LIST];
  float found;
};

// Where the sum of the weights in descending order, on top of `base`, first reaches `target`: the weight there, or `none`. The
// cluster's lists (of turn `turn`) hold `n` <= NUCLEUS_LIST of them, which every CTA sorts for itself: equal weights are
// alike, so neither the order within a list nor anything else of the launch shows in the result.
template <int CTAS>
__device__ __forceinline__ float nucleus_from_lists(NucleusShared& sh, int turn, int n, float base, float target, float none) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float v = 0.f;
  if constexpr (CTAS == 1) {
    if (tid < n) v = sh.list[tid];
  } else {
    cg::cluster_group cluster = cg::this_cluster();
    int count[CTAS], at = tid;
#pragma unroll
    for (int r = 0; r < CTAS; ++r) count[r] = *cluster.map_shared_rank(&sh.listed[turn], r);
#pragma unroll
    for (int r = 0; r < CTAS; ++r) {
      if (at >= 0 && at < count[r]) v = *cluster.map_shared_rank(&sh.list[at], r);
      at -= count[r];
    }
  }
  int size = 32;
  while (size < n) size <<= 1;
  for (int k = 2; k <= size; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {      // bitonic, descending
      float other;
      if (j >= 32) {
        __syncthreads();
        sh.sorted[tid] = v;
        __syncthreads();
        other = sh.sorted[tid ^ j];
      } else {
        other = __shfl_xor_sync(0xffffffffu, v, j);
      }
      v = (((tid & j) == 0) == ((tid & k) == 0)) ? fmaxf(v, other) : fminf(v, other);
    }
  float sum = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float below = __shfl_up_sync(0xffffffffu, sum, o);
    if (lane >= o) sum += below;
  }
  if (lane == 31) sh.scratch[warp] = sum;
  if (tid == 0) sh.found = none;
  __syncthreads();
  float before = lane < warp ? sh.scratch[lane] : 0.f;      // of the warps in front
  before = base + warp_sum(before);
  const unsigned reached = __ballot_sync(0xffffffffu, tid < n && !(before + sum < target));
  __syncthreads();
  if (lane == 0) sh.scratch[warp] = reached ? 1.f : 0.f;
  __syncthreads();
  const unsigned warps = __ballot_sync(0xffffffffu, sh.scratch[lane] != 0.f);
  if (warps && warp == __ffs(warps) - 1 && lane == __ffs(reached) - 1) sh.found = v;
  __syncthreads();
  return sh.found;
}

// COUNT values per CTA over the cluster: their sums in the order of the CTAs, or the largest. `turn` alternates from
// call to call, so that one barrier of all CTAs a call is enough.
template <int CTAS, int COUNT, bool MAX>
__device__ __forceinline__ const float* nucleus_exchange(NucleusShared& sh, int turn) {
  if constexpr (CTAS == 1) {
    __syncthreads();
    return sh.mine[turn];
  } else {
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();                       // everyone's `mine` of this turn is written
    if (threadIdx.x < COUNT) {
      float v[CTAS];
#pragma unroll
      for (int r = 0; r < CTAS; ++r) v[r] = *cluster.map_shared_rank(&sh.mine[turn][threadIdx.x], r);
      float t = v[0];
#pragma unroll
      for (int r = 1; r < CTAS; ++r) t = MAX ? fmaxf(t, v[r]) : t + v[r];
      sh.whole[turn][threadIdx.x] = t;
    }
    __syncthreads();
    return sh.whole[turn];
  }
}

// HELD: weights a thread keeps in registers, 0: they are read and raised again in every pass.
template <int CTAS, int HELD>
__device__ __forceinline__ float nucleus_threshold(const float* __restrict__ l, int vocab, int begin, int end, float inv_t, float top_p,
                                                   float& row_max, NucleusShared& sh) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float e[HELD ? HELD : 1];
  float mx = -INFINITY;
  if (HELD) {
#pragma unroll
    for (int j = 0; j < HELD; ++j) {
      const int i = begin + tid + j * SM_THREADS;
      e[j] = i < end ? l[i] : -INFINITY;
      mx = fmaxf(mx, scaled(e[j], inv_t));
    }
  } else {
    for (int i = begin + tid; i < end; i += SM_THREADS) mx = fmaxf(mx, scaled(l[i], inv_t));
  }
  mx = block_max(mx, sh.scratch);
  if (tid == 0) sh.mine[0][0] = mx;
  mx = nucleus_exchange<CTAS, 1, true>(sh, 0)[0];
  row_max = mx;

  float z = 0.f;
  if (HELD) {
#pragma unroll
    for (int j = 0; j < HELD; ++j) {
      e[j] = begin + tid + j * SM_THREADS < end ? weight_of(e[j], inv_t, mx) : 0.f;     // 0 is above no threshold
      z += e[j];
    }
  } else {
    for (int i = begin + tid; i < end; i += SM_THREADS) z += weight_of(l[i], inv_t, mx);
  }
  z = block_sum(z, sh.scratch);
  if (tid == 0) { sh.mine[1][0] = z; sh.listed[0] = sh.listed[1] = 0; }
  const float all = nucleus_exchange<CTAS, 1, false>(sh, 1)[0], target = top_p * all;
  if (!(target == target)) return 1.f;        // no threshold's sum is below it

  uint32_t lo = 0u, hi = 0x3f800000u;
  // A threshold's sum is short of the whole by at most the threshold times the number of tokens, so it reaches the target at
  // half of (1 - top_p) times their mean weight, unless 1 - top_p is a matter of rounding.
  if (1.f - top_p > 1e-4f) lo = __float_as_uint(fminf(0.5f * (1.f - top_p) * all / (float)vocab, 1.f));
  int turn = 0;
  bool open = true;                     // whether a weight of this warp may lie between the bounds
  float base = 0.f;                     // the sum above `hi`
  auto list_between = [&](int which) {
    if constexpr (HELD > 0) {
      // weights at or below float(lo) count for no threshold left, those above float(hi) for each of them
      const float low = __uint_as_float(lo), high = __uint_as_float(hi);
      if (!open) return;
      int between = 0;
      float above = 0.f;
#pragma unroll
      for (int j = 0; j < HELD; ++j) {
        between += e[j] > low && e[j] <= high ? 1 : 0;
        if (e[j] > high) above += e[j];
      }
      const int of_warp = __reduce_add_sync(0xffffffffu, between);
      open = of_warp != 0;
      if (!open) {
        above = warp_sum(above);
        if (lane < NUCLEUS_WAYS - 1) sh.by_warp[lane][warp] = above;
        return;
      }
      int at = 0;
      if (lane == 0) at = atomicAdd(&sh.listed[which], of_warp);
      at = __shfl_sync(0xffffffffu, at, 0);
      if (at + of_warp > NUCLEUS_LIST) return;
      int in_front = between;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int below = __shfl_up_sync(0xffffffffu, in_front, o);
        if (lane >= o) in_front += below;
      }
      at += in_front - between;
#pragma unroll
      for (int j = 0; j < HELD; ++j)
        if (e[j] > low && e[j] <= high) sh.list[at++] = e[j];
    }
  };
  list_between(0);
  while (lo < hi) {
    if (open) {        // else the warp's sums, the same for every threshold left, are where it has put them
      float t[NUCLEUS_WAYS - 1], mass[NUCLEUS_WAYS - 1];
#pragma unroll
      for (int q = 0; q < NUCLEUS_WAYS - 1; ++q) {
        t[q] = __uint_as_float(lo + (uint32_t)(((unsigned long long)(hi - lo) * (q + 1)) / NUCLEUS_WAYS));
        mass[q] = 0.f;
      }
      if (HELD) {
#pragma unroll
        for (int j = 0; j < HELD; ++j)
#pragma unroll
          for (int q = 0; q < NUCLEUS_WAYS - 1; ++q)
            if (e[j] > t[q]) mass[q] += e[j];
      } else {
        for (int i = begin + tid; i < end; i += SM_THREADS) {
          const float v = weight_of(l[i], inv_t, mx);
#pragma unroll
          for (int q = 0; q < NUCLEUS_WAYS - 1; ++q)
            if (v > t[q]) mass[q] += v;
        }
      }
#pragma unroll
      for (int q = 0; q < NUCLEUS_WAYS - 1; ++q) {
        const float v = warp_sum(mass[q]);
        if (lane == 0) sh.by_warp[q][warp] = v;
      }
    }
    __syncthreads();
    if (warp < NUCLEUS_WAYS - 1) {
      const float v = warp_sum(sh.by_warp[warp][lane]);
      if (lane == 0) sh.mine[turn][warp] = v;
    } else if (tid == SM_THREADS - 1) {
      sh.mine[turn][NUCLEUS_WAYS - 1] = (float)sh.listed[turn];
      sh.listed[turn ^ 1] = 0;
    }
    const float* whole = nucleus_exchange<CTAS, NUCLEUS_WAYS, false>(sh, turn);
    if (HELD && whole[NUCLEUS_WAYS - 1] <= (float)NUCLEUS_LIST)
      return nucleus_from_lists<CTAS>(sh, turn, (int)whole[NUCLEUS_WAYS - 1], base, target, __uint_as_float(lo));
    // sums of the same terms in the same order grow as the threshold falls: the first one below the target ends the search
    uint32_t below = lo, next = hi;
    bool found = false;
#pragma unroll
    for (int q = 0; q < NUCLEUS_WAYS - 1; ++q) {
      const uint32_t mid = lo + (uint32_t)(((unsigned long long)(hi - lo) * (q + 1)) / NUCLEUS_WAYS);
      if (!found) {
        if (whole[q] < target) { next = mid; base = whole[q]; found = true; }
        else below = mid + 1u;
      }
    }
    lo = below;
    hi = next;
    turn ^= 1;
    list_between(turn);
  }
  return __uint_as_float(lo);
}

// CTAS > 0: some rows have a top-p; the chunks of a row are the CTAS CTAs of a cluster.
template <int CTAS, int HELD>
__global__ void __launch_bounds__(SM_THREADS) sample_kernel(const float* __restrict__ logits, int vocab,
                                                            const float* __restrict__ temperature,
                                                            const float* __restrict__ top_p,
                                                            const long long* __restrict__ seeds,
                                                            const long long* __restrict__ draws,
                                                            int* __restrict__ out, int chunks,
                                                            const int* __restrict__ status_in,
                                                            int* __restrict__ status_out) {
  __shared__ Best bscratch[32];
  __shared__ int is_last;
  pdl_trigger();
  pdl_wait();
  const int row = blockIdx.x, chunk = blockIdx.y;
  // the step's error word (set by a kernel whose bounded wait ran out) travels to the host with the tokens
  if (status_out != nullptr && row == 0 && chunk == 0 && threadIdx.x == 0) *status_out = status_in ? *status_in : 0;
  const float* l = logits + (size_t)row * vocab;
  const float temp = temperature ? temperature[row] : 0.f;
  const float tp = (top_p && temp > 0.f) ? top_p[row] : 1.f;
  uint32_t k0 = 0, k1 = 0, d0 = 0, d1 = 0;
  if (temp > 0.f) {
    k0 = (uint32_t)(seeds[row] & 0xffffffffll); k1 = (uint32_t)((unsigned long long)seeds[row] >> 32);
    d0 = (uint32_t)(draws[row] & 0xffffffffll); d1 = (uint32_t)((unsigned long long)draws[row] >> 32);
  }
  int per = (vocab + chunks - 1) / chunks;
  per = (per + 3) & ~3;
  const int begin = chunk * per, end = min(vocab, begin + per);     // empty behind the last token
  float mx = 0.f, threshold = 0.f;
  if constexpr (CTAS > 0) if (tp < 1.f) {
    __shared__ NucleusShared sh;
    threshold = nucleus_threshold<CTAS, HELD>(l, vocab, begin, end, 1.f / temp, tp, mx, sh);
  }

  // ---- this CTA's chunk, then one CTA picks among the chunks
  Best best = scan_range(l, begin, end, temp, mx, threshold, k0, k1, d0, d1);
  best = block_best(best, bscratch);
  if constexpr (CTAS > 1) {
    // the first CTA of the cluster, through distributed shared memory: launches on several streams share nothing
    __shared__ Best mine;
    cg::cluster_group cluster = cg::this_cluster();
    if (threadIdx.x == 0) mine = best;
    cluster.sync();
    if (chunk == 0 && threadIdx.x == 0) {
      Best b[CTAS];
#pragma unroll
      for (int r = 0; r < CTAS; ++r) b[r] = *cluster.map_shared_rank(&mine, r);
#pragma unroll
      for (int r = 1; r < CTAS; ++r) b[0] = better(b[0], b[r]);
      out[row] = b[0].i < 0 ? 0 : b[0].i;
    }
    cluster.sync();          // nobody leaves while its winner (or its last sums of the search) may still be read
    return;
  }
  if (chunks == 1) {
    if (threadIdx.x == 0) out[row] = best.i < 0 ? 0 : best.i;
    return;
  }
  if (threadIdx.x == 0) g_chunk_best[row * SM_MAX_CHUNKS + chunk] = best;
  if (!cta_arrives_last(&g_row_arrivals[row], (unsigned int)chunks, &is_last)) return;
  if (threadIdx.x < 32) {
    // one lane per chunk (chunks <= 32): independent loads, then a warp reduction
    Best b;
    b.v = 0.f; b.i = -1;
    if ((int)threadIdx.x < chunks) {
      b.v = __ldcg(&g_chunk_best[row * SM_MAX_CHUNKS + threadIdx.x].v);
      b.i = __ldcg(&g_chunk_best[row * SM_MAX_CHUNKS + threadIdx.x].i);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      Best y;
      y.v = __shfl_xor_sync(0xffffffffu, b.v, o);
      y.i = __shfl_xor_sync(0xffffffffu, b.i, o);
      b = better(b, y);
    }
    if (threadIdx.x == 0) out[row] = b.i < 0 ? 0 : b.i;
  }
}

}  // namespace ts

using namespace ts;

// temperature/top_p/seeds/draws may all be null for an all-greedy batch. status_out (optional)
// receives *status_in (0 if that is null): the device word that kernels with bounded waits set
// when a wait ran out, so that one copy brings the tokens and the step's status to the host.
extern "C" int ts_sample(const float* logits, int num_rows, int vocab, const float* temperature,
                         const float* top_p, const long long* seeds, const long long* draws, int* out,
                         const int* status_in, int* status_out, cudaStream_t stream) {
  if (num_rows <= 0) return 0;
  if (vocab <= 0 || num_rows > SM_MAX_ROWS) return TS_ERR_BAD_ARGUMENT;
  if (temperature != nullptr && (seeds == nullptr || draws == nullptr)) return TS_ERR_BAD_ARGUMENT;
  if (temperature != nullptr && top_p != nullptr) {
    // As few CTAs a row as hold its weights in registers: one CTA fits an SM, so eight let 18 rows run at once, and what a
    // pass costs besides its tokens (the cluster's barrier and exchange) is paid by each. The number of rows has no say: a
    // row's sums are the same in any batch.
    constexpr int one = NUCLEUS_HELD * SM_THREADS;
#define TS_NUCLEUS(CTAS_, HELD_)                                                                                                    \
    return launch_cluster(sample_kernel<CTAS_, HELD_>, dim3(num_rows, CTAS_), SM_THREADS, 0, stream, dim3(1, CTAS_), logits, vocab, \
                          temperature, top_p, seeds, draws, out, CTAS_, status_in, status_out)
    if (vocab <= one) {
      auto kernel = vocab <= NUCLEUS_HELD_SMALL * SM_THREADS ? sample_kernel<1, NUCLEUS_HELD_SMALL> : sample_kernel<1, NUCLEUS_HELD>;
      return launch(kernel, dim3(num_rows), SM_THREADS, 0, stream, logits, vocab, temperature, top_p, seeds, draws, out, 1, status_in,
                    status_out);
    }
    if (vocab <= 2 * one) TS_NUCLEUS(2, NUCLEUS_HELD);
    if (vocab <= 4 * one) TS_NUCLEUS(4, NUCLEUS_HELD);
    if (vocab <= 8 * one) TS_NUCLEUS(8, NUCLEUS_HELD);
    TS_NUCLEUS(8, 0);
#undef TS_NUCLEUS
  }
  // as many CTAs as run at once (two of 1024 threads per SM), never a partly filled second
  // round, each with at least a few thousand tokens
  int chunks = (148 * 2) / num_rows;
  const int most = (vocab + 4095) / 4096;
  if (chunks > most) chunks = most;
  if (chunks > SM_MAX_CHUNKS) chunks = SM_MAX_CHUNKS;
  if (chunks < 1) chunks = 1;
  return launch(sample_kernel<0, 0>, dim3(num_rows, chunks), SM_THREADS, 0, stream, logits, vocab, temperature, top_p,
                seeds, draws, out, chunks, status_in, status_out);
}
