// Paged attention on CUDA cores (kernel templates and their launch helpers), for float and bf16: the true 32-bit path of the engine and
// the fallback for head sizes the tensor-core kernels do not take.
//
// Math (upstream src/tinyserve/attention.py:89-111): s = scale * q.k over head_dim in 32-bit,
// causal mask (key position <= query position; optionally > query position - window, or
// below `keep_first`: the first positions that a window never drops; or in the query's own chunk),
// softmax in 32-bit (online, base 2), o = sum p v in 32-bit, cast once to the output type.
// Query head h reads kv head h / (num_heads / num_kv_heads).
//
//  * prefill kernel: one CTA per (tile of 16 or 32 queries of one request, query head); keys and
//    values are staged through shared memory in tiles of 32 (after upstream
//    src/tinyserve/triton_prefill.py:50-125, which tiles the same way over the paged cache).
//  * decode kernel: one CTA per (request, kv head, split of the keys); a group of lanes reads
//    one key with 16-byte loads, all query heads of the group share each key and value; the
//    CTA that finishes last merges the splits (the split-K scheme is upstream's,
//    src/tinyserve/triton_attention.py:243-327, which merges in a second kernel).
// Keys outside a request's own range are never loaded: their scores are -inf and their values
// zero, so whatever lies in pages of other requests cannot reach the result.
#pragma once
#include "attention.cuh"

namespace ts {

constexpr float NEG_INF = -INFINITY;

// =============================================================== prefill (tiled)
// What bounds it at the sizes it serves (the 32-bit path's prompts, odd head sizes): the serial chain of a CTA's key tiles.
// So the operands lie in shared memory in rows of whole 16-byte words and are read four elements at a time (scalar reads
// cost six shared-memory instructions for eight multiply-adds), float tiles come by cp.async into the second buffer
// while the first one is worked on, and a step with few CTAs is cut into tiles of 16 queries instead of 32. Whatever the
// cut, a row's scores are one chain over the head's elements, its sums go over the keys in order and are rescaled every
// 32 keys, so its result does not depend on the batch. B200, float, 16 / 8 heads of 128, staged and multiplied element by
// element / now: 45 tokens 24 / 15 us, 300 tokens 119 / 80, 64 tokens at 2,000 positions 615 / 358, 2,000 tokens 1,290 / 1,098.
constexpr int PF_TK = 32;       // keys per tile
constexpr int PF_THREADS = 128;

__device__ __forceinline__ void pf_copy16(float* dst, const void* src, bool ok) {
  const unsigned int d = (unsigned int)__cvta_generic_to_shared(dst);
  const int n = ok ? 16 : 0;     // zeros where the key is not visible
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

// Shared memory in floats: queries [TQ][DS], `buffers` x (keys [TK][DS], values [TK][VS]), scores [TQ][TK + 4], 3 row arrays.
// DS, VS: the head sizes up to a multiple of 4, plus one 16-byte word (rows that eight neighbouring threads read start in
// eight different groups of banks).
__host__ __device__ __forceinline__ int pf_stride(int d) { return (d + 3) / 4 * 4 + 4; }
constexpr int PF_SS = PF_TK + 4;
static inline size_t pf_smem(int tq, int D, int DV, int buffers) {
  return sizeof(float) * ((size_t)tq * pf_stride(D) + (size_t)buffers * PF_TK * (pf_stride(D) + pf_stride(DV)) + (size_t)tq * PF_SS + 3 * tq);
}

// TQ = queries per CTA (16 or 32); QJ = groups of 64 value columns (a thread owns four neighbouring ones of each).
template <typename T, int TQ, int QJ>
__global__ void __launch_bounds__(PF_THREADS) prefill_attn_kernel(AttnArgs a, int buffers) {
  constexpr int RT = TQ / 8;                    // rows a thread owns
  extern __shared__ __align__(16) float smem[];
  const int D = a.head_dim;
  const int DV = a.v_head_dim ? a.v_head_dim : D;   // values may have a head size of their own
  const int DS = pf_stride(D), VS = pf_stride(DV);
  float* Qs = smem;                             // [TQ][DS]  pre-scaled queries
  float* tiles = Qs + TQ * DS;
  const int tile_floats = PF_TK * (DS + VS);
  float* Ss = tiles + buffers * tile_floats;    // [TQ][PF_SS]
  float* row_m = Ss + TQ * PF_SS;               // [TQ]
  float* row_l = row_m + TQ;                    // [TQ]
  float* row_c = row_l + TQ;                    // [TQ] correction factor of this tile

  pdl_trigger();
  pdl_wait();
  const int seq = a.seq_ids[blockIdx.y];
  const int head = blockIdx.z;
  const int kvh = head / (a.num_heads / a.num_kv_heads);
  const int row0 = a.cu_q[seq];
  const int n = a.cu_q[seq + 1] - row0;
  const int q0 = blockIdx.x * TQ;
  if (q0 >= n) return;
  const int ctx = a.ctx_lens[seq];
  const int first_pos = ctx - n;                // position of the request's first new token
  const int nq = min(TQ, n - q0);
  const int* table = a.block_tables + (size_t)seq * a.table_width;
  const T* q = (const T*)a.q;
  const T* kc = (const T*)a.k_cache;
  const T* vc = (const T*)a.v_cache;
  const int tid = threadIdx.x;

  const int qpos_first = first_pos + q0;
  const int qpos_last = first_pos + q0 + nq - 1;
  const int k_lo = first_visible(qpos_first, a);
  const int k_begin = (k_lo / PF_TK) * PF_TK;
  // with kept first positions the tiles below the window that hold any of them come first
  const int kept = (a.window > 0) ? min(a.keep_first, k_lo) : 0;
  const int kept_end = min(k_begin, ((kept + PF_TK - 1) / PF_TK) * PF_TK);
  constexpr int VEC = Vec<T>::N;
  const bool vec_ok = (D % VEC == 0) && (DV % VEC == 0);

  // Keys and values k0 .. k0 + TK - 1 into a buffer (zeros outside the request's visible range and in the padding columns).
  // Four threads a key: one look-up in the block table each, then nothing but copies.
  const int skey = tid >> 2, spart = tid & 3;
  auto stage = [&](int k0, float* Ks) {
    const int kpos = k0 + skey;
    const bool ok = (kpos >= k_lo || kpos < kept) && kpos <= qpos_last;
    const size_t row = ok ? kv_row_of(table, kpos, kvh, a) : 0;
    auto copy = [&](const T* src, float* dst, int n) {      // n elements of a row; the thread's share of it
      if (vec_ok) {
#pragma unroll 4
        for (int c = spart * VEC; c < n; c += 4 * VEC) {
          if constexpr (VEC == 4) {
            pf_copy16(dst + c, src + c, ok);
          } else {
            float f[VEC];
            Vec<T> raw;
            if (ok) raw.load(src + c); else raw.zero();
            raw.unpack(f);
#pragma unroll
            for (int e = 0; e < VEC; e += 4) *reinterpret_cast<float4*>(dst + c + e) = make_float4(f[e], f[e + 1], f[e + 2], f[e + 3]);
          }
        }
      } else {
        // head sizes that are no multiple of a 16-byte vector: element by element, the padding included
        for (int c = spart; c < pf_stride(n) - 4; c += 4) dst[c] = ok && c < n ? to_float(src[c]) : 0.f;
      }
    };
    copy(kc + row * D, Ks + skey * DS, D);
    copy(vc + row * DV, Ks + PF_TK * DS + skey * VS, DV);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto next_tile = [&](int k0) { return (k0 + PF_TK == kept_end) ? k_begin : k0 + PF_TK; };

  int k0 = kept_end > 0 ? 0 : k_begin, turn = 0;
  stage(k0, tiles);
  {
    constexpr int TPR = PF_THREADS / TQ;        // threads per query row
    const int r = tid / TPR;
    const T* src = q + q_row_of(row0 + q0 + (r < nq ? r : 0), head, a) * D;
#pragma unroll 4
    for (int c = tid % TPR * 4; c < DS - 4; c += 4 * TPR) {
      float f[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int d = c + e;
        f[e] = r < nq && d < D && q_col_lives(head, d, D, a) ? to_float(src[d]) * a.scale_log2 : 0.f;
      }
      *reinterpret_cast<float4*>(Qs + r * DS + c) = make_float4(f[0], f[1], f[2], f[3]);
    }
  }
  if (tid < TQ) { row_m[tid] = NEG_INF; row_l[tid] = 0.f; }

  const int ty = tid >> 4, tx = tid & 15;       // 8 row groups x 16 column groups
  float4 acc[RT][QJ];
#pragma unroll
  for (int i = 0; i < RT; ++i)
#pragma unroll
    for (int j = 0; j < QJ; ++j) acc[i][j] = make_float4(0.f, 0.f, 0.f, 0.f);

  while (true) {
    const int k_next = next_tile(k0);
    const bool more = k_next <= qpos_last;
    const float* Ks = tiles + turn * tile_floats;
    const float* Vs = Ks + PF_TK * DS;
    // with two buffers the next tile is asked for now: its buffer was read before the barrier at the end of the last tile
    if (buffers == 2 && more) {
      stage(k_next, tiles + (turn ^ 1) * tile_floats);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    // ---- scores: thread (ty, tx) owns RT rows from ty * RT, keys tx and tx + 16
    float s[RT][2];
#pragma unroll
    for (int i = 0; i < RT; ++i) { s[i][0] = 0.f; s[i][1] = 0.f; }
#pragma unroll 4
    for (int d = 0; d < DS - 4; d += 4) {
      const float4 u = *reinterpret_cast<const float4*>(Ks + tx * DS + d);
      const float4 v = *reinterpret_cast<const float4*>(Ks + (tx + 16) * DS + d);
#pragma unroll
      for (int i = 0; i < RT; ++i) {
        const float4 x = *reinterpret_cast<const float4*>(Qs + (ty * RT + i) * DS + d);
        s[i][0] = fmaf(x.w, u.w, fmaf(x.z, u.z, fmaf(x.y, u.y, fmaf(x.x, u.x, s[i][0]))));
        s[i][1] = fmaf(x.w, v.w, fmaf(x.z, v.z, fmaf(x.y, v.y, fmaf(x.x, v.x, s[i][1]))));
      }
    }
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      const int r = ty * RT + i;
      const int qpos = first_pos + q0 + r;
      const int first = first_visible(qpos, a);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int kpos = k0 + tx + 16 * j;
        const bool ok = (r < nq) && (kpos <= qpos) && (kpos >= first || kpos < a.keep_first);
        Ss[r * PF_SS + tx + 16 * j] = ok ? s[i][j] : NEG_INF;
      }
    }
    __syncthreads();
    // ---- online softmax per row: 4 threads per row
    if (tid < 4 * TQ) {
      const int r = tid >> 2, part = tid & 3;
      float* srow = Ss + r * PF_SS;
      float mx = NEG_INF;
#pragma unroll
      for (int j = 0; j < PF_TK / 4; ++j) mx = fmaxf(mx, srow[part * (PF_TK / 4) + j]);
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      const float m_old = row_m[r];
      const float m_new = fmaxf(m_old, mx);
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < PF_TK / 4; ++j) {
        const int col = part * (PF_TK / 4) + j;
        const float sv = srow[col];
        const float p = (sv == NEG_INF) ? 0.f : exp2f(sv - m_new);
        srow[col] = p;
        sum += p;
      }
      sum += __shfl_xor_sync(0xffffffffu, sum, 1);
      sum += __shfl_xor_sync(0xffffffffu, sum, 2);
      __syncwarp();
      if (part == 0) {
        const float corr = (m_new == NEG_INF) ? 1.f : exp2f(m_old - m_new);  // m_old = -inf gives 0
        row_c[r] = corr;
        row_l[r] = row_l[r] * corr + sum;
        row_m[r] = m_new;
      }
    }
    __syncthreads();
    // ---- acc = acc * corr + P V: thread owns RT rows, columns 4 tx .. + 3 of every 64
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      const float corr = row_c[ty * RT + i];
#pragma unroll
      for (int j = 0; j < QJ; ++j) { acc[i][j].x *= corr; acc[i][j].y *= corr; acc[i][j].z *= corr; acc[i][j].w *= corr; }
    }
#pragma unroll 2
    for (int kk = 0; kk < PF_TK; kk += 4) {
      float p[RT][4];
#pragma unroll
      for (int i = 0; i < RT; ++i) {
        const float4 v = *reinterpret_cast<const float4*>(Ss + (ty * RT + i) * PF_SS + kk);
        p[i][0] = v.x; p[i][1] = v.y; p[i][2] = v.z; p[i][3] = v.w;
      }
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int j = 0; j < QJ; ++j) {
          if (4 * tx + 64 * j < DV) {
            const float4 vv = *reinterpret_cast<const float4*>(Vs + (kk + e) * VS + 4 * tx + 64 * j);
#pragma unroll
            for (int i = 0; i < RT; ++i) {
              acc[i][j].x = fmaf(p[i][e], vv.x, acc[i][j].x);
              acc[i][j].y = fmaf(p[i][e], vv.y, acc[i][j].y);
              acc[i][j].z = fmaf(p[i][e], vv.z, acc[i][j].z);
              acc[i][j].w = fmaf(p[i][e], vv.w, acc[i][j].w);
            }
          }
        }
    }
    if (!more) break;
    __syncthreads();       // this tile's keys, values and scores have been read by everyone
    if (buffers == 1) stage(k_next, tiles);
    else turn ^= 1;
    k0 = k_next;
  }
  T* out = (T*)a.out;
#pragma unroll
  for (int i = 0; i < RT; ++i) {
    const int r = ty * RT + i;
    if (r < nq) {
#pragma unroll
      for (int j = 0; j < QJ; ++j) {
        const float v[4] = {acc[i][j].x, acc[i][j].y, acc[i][j].z, acc[i][j].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int c = 4 * tx + 64 * j + e;
          if (c < DV)
            out[((size_t)(row0 + q0 + r) * a.num_heads + head) * DV + c] = from_float<T>(finish_row(v[e], row_l[r], row_m[r], a.sinks, head));
        }
      }
    }
  }
}

// ================================================================ decode (split-K)
// A CTA has eight warps, or four when there are this many CTAs, three an SM, to fill the machine (float, 12 / 3 heads of 64,
// 64 requests of 200 positions, 576 CTAs: 26 us with eight, 18 with four; 16 / 8 of 128, 16 of 1,000, 640 CTAs, 54 / 40; one
// of 500, 56 CTAs, 9.3 / 10.3).
constexpr int DC_MANY_CTAS = 444;
constexpr int DC_MAX_COUNTERS = 1 << 16;

// One arrival counter per (request, CTA row of the grid): the CTA that arrives last merges the
// key ranges. Counters are zero when the library is loaded and every merge puts its counter
// back to zero, so no launch ever has to clear them.
static __device__ unsigned int g_decode_counters[DC_MAX_COUNTERS];

// GT = query heads handled per CTA (a kv group is covered by ceil(G / GT) CTAs);
// LPK = lanes that share a key; CPL = 16-byte chunks of a key per lane; U = keys per lane group whose loads are in flight.
// Bound by its chain of latencies: block table, keys, the sums over the lanes of a key, the exponentials. Few lanes a key
// make few exchanges (three steps for four keys at once with LPK = 8, five for one with 32), and the number of lanes is
// known to the compiler so that the exchanges of all keys and heads overlap. Float, 16 / 8 heads of 128, 32 lanes a key and
// four warps / now: one request of 500 positions 21 / 9 us, 16 of 1,000 111 / 40; 32 / 8 heads, 64 of 200 95 / 54.
template <typename T, int GT, int CPL, int LPK, int U, int WARPS>
__global__ void __launch_bounds__(WARPS * 32) decode_attn_kernel(AttnArgs a, int passes) {
  constexpr int VEC = Vec<T>::N;
  constexpr int EPL = VEC * CPL;                 // elements of a key per lane
  extern __shared__ float smem[];                // [WARPS][GT][D + 2]
  __shared__ int is_last;
  pdl_trigger();
  const int D = a.head_dim;
  const int G = a.num_heads / a.num_kv_heads;
  const int si = blockIdx.x;
  const int kvh = blockIdx.y / passes;
  const int g0 = (blockIdx.y - kvh * passes) * GT;   // first head of the group this CTA handles
  const int ng = min(GT, G - g0);
  const int split = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane / LPK, lk = lane - sub * LPK;  // which key of the warp's batch, which lane of it
  constexpr int KPW = 32 / LPK;                       // keys per warp per batch
  const int chunks = D / VEC;
  pdl_wait();

  const int seq = a.seq_ids[si];
  const int ctx = a.ctx_lens[seq];
  const int qrow = a.cu_q[seq];
  const int lo = first_visible(ctx - 1, a);
  // the visible keys in one run of indices: the kept first positions below the window, then the window
  const int kept = min(a.keep_first, lo);
  const int gap = lo - kept;
  const int len = ctx - gap;
  const int per = (len + a.num_splits - 1) / a.num_splits;
  const int k_begin = split * per;
  const int k_end = min(len, k_begin + per);
  const int* table = a.block_tables + (size_t)seq * a.table_width;
  const T* kc = (const T*)a.k_cache;
  const T* vc = (const T*)a.v_cache;

  // this lane's share of every query head, pre-scaled
  float qreg[GT][EPL];
#pragma unroll
  for (int g = 0; g < GT; ++g)
#pragma unroll
    for (int c = 0; c < CPL; ++c) {
      const int chunk = lk + c * LPK;
      float f[VEC];
      if (g < ng && chunk < chunks && q_col_lives(kvh * G + g0 + g, chunk * VEC, D, a)) {
        Vec<T> v;
        v.load((const T*)a.q + q_row_of(qrow, kvh * G + g0 + g, a) * D + chunk * VEC);
        v.unpack(f);
      } else {
#pragma unroll
        for (int e = 0; e < VEC; ++e) f[e] = 0.f;
      }
#pragma unroll
      for (int e = 0; e < VEC; ++e) qreg[g][c * VEC + e] = f[e] * a.scale_log2;
    }

  float m[GT], l[GT], acc[GT][EPL];
#pragma unroll
  for (int g = 0; g < GT; ++g) {
    m[g] = NEG_INF;
    l[g] = 0.f;
#pragma unroll
    for (int e = 0; e < EPL; ++e) acc[g][e] = 0.f;
  }

  const int stride = WARPS * KPW * U;
  for (int base = k_begin + (warp * U) * KPW; base < k_end; base += stride) {
    // ---- all loads of this batch first: U keys and U values per lane group, kept packed
    Vec<T> kraw[U][CPL], vraw[U][CPL];
    bool valid[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int kidx = base + u * KPW + sub;
      valid[u] = kidx < k_end;
      size_t off = 0;
      if (valid[u]) off = kv_offset_of(table, kidx < kept ? kidx : kidx + gap, kvh, a);
#pragma unroll
      for (int c = 0; c < CPL; ++c) {
        const int chunk = lk + c * LPK;
        if (valid[u] && chunk < chunks) {
          kraw[u][c].load(kc + off + (size_t)chunk * VEC);
          vraw[u][c].load(vc + off + (size_t)chunk * VEC);
        } else {
          kraw[u][c].zero();
          vraw[u][c].zero();
        }
      }
    }
    // ---- scores
    float s[GT][U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float kf[EPL];
#pragma unroll
      for (int c = 0; c < CPL; ++c) kraw[u][c].unpack(&kf[c * VEC]);
#pragma unroll
      for (int g = 0; g < GT; ++g) {
        float d = 0.f;
#pragma unroll
        for (int e = 0; e < EPL; ++e) d = fmaf(qreg[g][e], kf[e], d);
        s[g][u] = d;
      }
    }
#pragma unroll
    for (int g = 0; g < GT; ++g)
#pragma unroll
      for (int u = 0; u < U; ++u) {
        float d = s[g][u];
#pragma unroll
        for (int o = LPK >> 1; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        s[g][u] = valid[u] ? d : NEG_INF;
      }
    // ---- online softmax, one rescale per batch
#pragma unroll
    for (int g = 0; g < GT; ++g) {
      float m_new = m[g];
#pragma unroll
      for (int u = 0; u < U; ++u) m_new = fmaxf(m_new, s[g][u]);
      const float corr = (m_new == NEG_INF) ? 1.f : exp2f(m[g] - m_new);   // m = -inf gives 0
      float psum = 0.f;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const float p = (s[g][u] == NEG_INF) ? 0.f : exp2f(s[g][u] - m_new);
        s[g][u] = p;
        psum += p;
      }
      l[g] = l[g] * corr + psum;
      m[g] = m_new;
#pragma unroll
      for (int e = 0; e < EPL; ++e) acc[g][e] *= corr;
    }
    // ---- values
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float vf[EPL];
#pragma unroll
      for (int c = 0; c < CPL; ++c) vraw[u][c].unpack(&vf[c * VEC]);
#pragma unroll
      for (int g = 0; g < GT; ++g)
#pragma unroll
        for (int e = 0; e < EPL; ++e) acc[g][e] = fmaf(s[g][u], vf[e], acc[g][e]);
    }
  }

  // ---- merge the lane groups of a warp (lanes with equal lk hold the same elements)
#pragma unroll
  for (int o = LPK; o < 32; o <<= 1) {
#pragma unroll
    for (int g = 0; g < GT; ++g) {
      const float m2 = __shfl_xor_sync(0xffffffffu, m[g], o);
      const float l2 = __shfl_xor_sync(0xffffffffu, l[g], o);
      const float mn = fmaxf(m[g], m2);
      const float c1 = (mn == NEG_INF) ? 1.f : exp2f(m[g] - mn);
      const float c2 = (mn == NEG_INF) ? 1.f : exp2f(m2 - mn);
      l[g] = l[g] * c1 + l2 * c2;
#pragma unroll
      for (int e = 0; e < EPL; ++e) {
        const float a2 = __shfl_xor_sync(0xffffffffu, acc[g][e], o);
        acc[g][e] = acc[g][e] * c1 + a2 * c2;
      }
      m[g] = mn;
    }
  }
  // ---- merge the warps through shared memory
  const int WS = D + 2;
  if (sub == 0) {
#pragma unroll
    for (int g = 0; g < GT; ++g) {
      float* w = smem + ((size_t)warp * GT + g) * WS;
#pragma unroll
      for (int c = 0; c < CPL; ++c) {
        const int chunk = lk + c * LPK;
        if (chunk < chunks)
#pragma unroll
          for (int e = 0; e < VEC; ++e) w[chunk * VEC + e] = acc[g][c * VEC + e];
      }
      if (lk == 0) { w[D] = m[g]; w[D + 1] = l[g]; }
    }
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < ng * D; idx += WARPS * 32) {
    const int g = idx / D, d = idx - g * D;
    float mm = NEG_INF;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) mm = fmaxf(mm, smem[((size_t)w * GT + g) * WS + D]);
    float num = 0.f, den = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const float* ws = smem + ((size_t)w * GT + g) * WS;
      const float c = (ws[D] == NEG_INF) ? 0.f : exp2f(ws[D] - mm);
      num += ws[d] * c;
      den += ws[D + 1] * c;
    }
    const int head = kvh * G + g0 + g;
    if (a.num_splits == 1) {
      ((T*)a.out)[((size_t)qrow * a.num_heads + head) * D + d] = from_float<T>(finish_row(num, den, mm, a.sinks, head));
    } else {
      const size_t pidx = ((size_t)si * a.num_heads + head) * a.num_splits + split;
      a.part_acc[pidx * D + d] = num;
      if (d == 0) { a.part_ml[pidx * 2] = mm; a.part_ml[pidx * 2 + 1] = den; }
    }
  }
  if (a.num_splits == 1) return;

  // ---- the CTA that arrives last for this (request, heads) merges the ranges
  unsigned int* counter = &g_decode_counters[((size_t)si * gridDim.y + blockIdx.y) % DC_MAX_COUNTERS];
  if (!cta_arrives_last(counter, (unsigned int)a.num_splits, &is_last)) return;
  merge_splits<T>(a, si, qrow, kvh * G + g0, ng, smem);
}

template <typename T, int TQ, int QJ>
static int launch_prefill_tq(const AttnArgs& a, int max_query_len, cudaStream_t stream) {
  const int D = a.head_dim, DV = a.v_head_dim ? a.v_head_dim : D;
  int buffers = sizeof(T) == 4 ? 2 : 1;       // only float tiles come asynchronously
  if (pf_smem(TQ, D, DV, buffers) > 200 * 1024) buffers = 1;
  const size_t smem = pf_smem(TQ, D, DV, buffers);
  auto kern = prefill_attn_kernel<T, TQ, QJ>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  dim3 grid((max_query_len + TQ - 1) / TQ, a.num_seqs, a.num_heads);
  return launch(kern, grid, PF_THREADS, smem, stream, a, buffers);
}

template <typename T, int QJ>
static int launch_prefill_qj(const AttnArgs& a, int max_query_len, cudaStream_t stream) {
  // tiles of 16 queries while those of 32 leave SMs without a CTA (the work per query is then larger, but more of it at once)
  const long long ctas = (long long)((max_query_len + 31) / 32) * a.num_seqs * a.num_heads;
  return ctas < 148 ? launch_prefill_tq<T, 16, QJ>(a, max_query_len, stream) : launch_prefill_tq<T, 32, QJ>(a, max_query_len, stream);
}

template <typename T>
static int launch_prefill(const AttnArgs& a, int max_query_len, cudaStream_t stream) {
  const int qj = ((a.v_head_dim ? a.v_head_dim : a.head_dim) + 63) / 64;
  if (qj <= 1) return launch_prefill_qj<T, 1>(a, max_query_len, stream);
  if (qj <= 2) return launch_prefill_qj<T, 2>(a, max_query_len, stream);
  return launch_prefill_qj<T, 4>(a, max_query_len, stream);
}

template <typename T, int GT, int CPL, int LPK, int WARPS>
static int launch_decode_warps(const AttnArgs& a, int passes, cudaStream_t stream) {
  constexpr int U = CPL >= 8 ? 1 : CPL >= 4 ? 2 : (CPL == 1 && GT <= 4) ? 8 : 4;
  // the warps' sums; the merge of the ranges keeps its (max, sum) pairs in the same memory
  const size_t sums = (size_t)WARPS * GT * (a.head_dim + 2), pairs = (size_t)GT * a.num_splits * 2;
  const size_t smem = sizeof(float) * (sums > pairs ? sums : pairs);
  auto kern = decode_attn_kernel<T, GT, CPL, LPK, U, WARPS>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  dim3 grid(a.num_seqs, a.num_kv_heads * passes, a.num_splits);
  return launch(kern, grid, WARPS * 32, smem, stream, a, passes);
}

template <typename T, int GT, int CPL, int LPK>
static int launch_decode_gc(const AttnArgs& a, cudaStream_t stream) {
  const int G = a.num_heads / a.num_kv_heads;
  const int passes = (G + GT - 1) / GT;
  const long long rows = (long long)a.num_seqs * a.num_kv_heads * passes;
  if (rows > DC_MAX_COUNTERS && a.num_splits > 1) return TS_ERR_UNSUPPORTED;
  return rows * a.num_splits >= DC_MANY_CTAS ? launch_decode_warps<T, GT, CPL, LPK, 4>(a, passes, stream)
                                             : launch_decode_warps<T, GT, CPL, LPK, 8>(a, passes, stream);
}

template <typename T>
static int launch_decode(const AttnArgs& a, cudaStream_t stream) {
  constexpr int VEC = Vec<T>::N;
  const int chunks = a.head_dim / VEC;
  const int G = a.num_heads / a.num_kv_heads;
  if (chunks > 64) return TS_ERR_UNSUPPORTED;
  // Lanes a key and 16-byte chunks a lane: few lanes make few exchanges, but each holds its elements of every head's query
  // and sum, and too many of them leave no registers for keys in flight and no room for CTAs (float, 4 / 2 heads of 256, 16
  // requests of 1,000 positions: 8 lanes 43 us, 16 lanes 25; 32 / 8 of 128, 64 of 200: 32 lanes 113, 16 lanes 82; bf16, 16 / 2
  // of 256, 16 of 1,000, eight heads a CTA: 16 lanes 119, 32 lanes 81).
  if (G <= 2) {
#define TS_DECODE_CASE(GT_)                                                                \
    if (chunks <= 4) return launch_decode_gc<T, GT_, 1, 4>(a, stream);                     \
    if (chunks <= 8) return launch_decode_gc<T, GT_, 1, 8>(a, stream);                     \
    if (chunks <= 16) return launch_decode_gc<T, GT_, 2, 8>(a, stream);                    \
    if constexpr (VEC == 4) {                                                              \
      if (chunks <= 32) return launch_decode_gc<T, GT_, 4, 8>(a, stream);                  \
      return launch_decode_gc<T, GT_, 4, 16>(a, stream);                                   \
    } else {                                                                               \
      if (chunks <= 32) return launch_decode_gc<T, GT_, 2, 16>(a, stream);                 \
    }
    if (G == 1) { TS_DECODE_CASE(1); return TS_ERR_UNSUPPORTED; }
    TS_DECODE_CASE(2);
    return TS_ERR_UNSUPPORTED;
#undef TS_DECODE_CASE
  }
#define TS_DECODE_CASE(GT_)                                                   \
  if (chunks <= 4) return launch_decode_gc<T, GT_, 1, 4>(a, stream);                           \
  if (chunks <= 8) return launch_decode_gc<T, GT_, 1, 8>(a, stream);                           \
  if (chunks <= 16) return launch_decode_gc<T, GT_, GT_ == 4 ? 2 : 1, GT_ == 4 ? 8 : 16>(a, stream);   \
  if constexpr (VEC == 4 || GT_ == 4) {                                                        \
    if (chunks <= 32) return launch_decode_gc<T, GT_, 2, 16>(a, stream);                       \
  } else {                                                                                     \
    if (chunks <= 32) return launch_decode_gc<T, GT_, 1, 32>(a, stream);                       \
  }                                                                                            \
  if constexpr (VEC == 4) return launch_decode_gc<T, GT_, 2, 32>(a, stream)
  if (G <= 4) { TS_DECODE_CASE(4); return TS_ERR_UNSUPPORTED; }
  TS_DECODE_CASE(8);
#undef TS_DECODE_CASE
  return TS_ERR_UNSUPPORTED;
}

}  // namespace ts

