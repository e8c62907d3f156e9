// What the scans over chunks of 64 tokens share (state_space_chunks.cu, mlstm_chunks.cu): 32-bit products of register tiles
// out of shared memory, and the loads of their operands.
//
// Chunks are numbered over the whole step, request b's from cu_q[b] / 64 + b on (gaps of at most one), so scratch and
// grid follow the step's tokens, however unequal the requests are; a request of one token costs one chunk of one row.
#pragma once
#include "common.cuh"

namespace ts {

constexpr int SC_Q = 64;              // tokens of a chunk
constexpr int SC_V = 64;              // value columns of a CTA
constexpr int SC_LD = SC_Q + 4;       // row of a tile whose fast index is the token (16-byte aligned, spread over the banks)
constexpr int SC_MAX_STATE = 128;

// The request and the tokens of chunk g of the step; false for a number that belongs to no chunk.
__device__ __forceinline__ bool find_chunk(const int* cu_q, int num_seqs, int g, int& t0, int& nt, int* seq = nullptr) {
  int lo = 0, hi = num_seqs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (cu_q[mid] / SC_Q + mid <= g) lo = mid; else hi = mid - 1;
  }
  const int start = cu_q[lo], end = cu_q[lo + 1];
  t0 = start + (g - (start / SC_Q + lo)) * SC_Q;
  nt = min(SC_Q, end - t0);
  if (seq) *seq = lo;
  return nt > 0;
}

// acc[4 A][4] += A^T B over k rows: A's rows hold the 4 A-wide operand (row `lda` floats, this thread's part from `ar`), B's
// the 4-wide one. Both 16-byte aligned.
template <int A>
__device__ __forceinline__ void tile_product(float (&acc)[4 * A][4], const float* ar, int lda, const float* br, int ldb, int k) {
#pragma unroll 4
  for (int i = 0; i < k; ++i) {
    const float4 b = *reinterpret_cast<const float4*>(br + i * ldb);
#pragma unroll
    for (int q = 0; q < A; ++q) {
      const float4 a = *reinterpret_cast<const float4*>(ar + i * lda + 4 * q);
      const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        acc[4 * q + r][0] = fmaf(av[r], b.x, acc[4 * q + r][0]);
        acc[4 * q + r][1] = fmaf(av[r], b.y, acc[4 * q + r][1]);
        acc[4 * q + r][2] = fmaf(av[r], b.z, acc[4 * q + r][2]);
        acc[4 * q + r][3] = fmaf(av[r], b.w, acc[4 * q + r][3]);
      }
    }
  }
}

// The same, the terms added up 16 at a time and then block by block: short chains, and errors as small as those of a scan whose
// threads each add up a few rows.
template <int A>
__device__ __forceinline__ void tile_product_in_blocks(float (&acc)[4 * A][4], const float* ar, int lda, const float* br, int ldb, int k) {
  for (int i = 0; i < k; i += 16) {
    float part[4 * A][4] = {};
    tile_product<A>(part, ar + i * lda, lda, br + i * ldb, ldb, min(16, k - i));
#pragma unroll
    for (int r = 0; r < 4 * A; ++r)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[r][j] += part[r][j];
  }
}

// Loads in flight per thread before the first is stored to shared memory: one after the other each would wait for memory.
constexpr int SC_LOADS = 8;

// [nt rows of `width`] -> tile [SC_Q][ld], zero past the edges; four columns an access where the source allows it.
template <typename T>
__device__ __forceinline__ void load_rows(const T* src, int stride, int rows, int width, bool vec, float* dst, int ld, int cols,
                                          int total_rows, int tid, int threads) {
  const int quads = cols / 4, total = total_rows * quads;
  for (int base = tid; base < total; base += threads * SC_LOADS) {
    float4 v[SC_LOADS];
#pragma unroll
    for (int u = 0; u < SC_LOADS; ++u) {
      const int idx = base + u * threads, r = idx / quads, c = (idx - r * quads) * 4;
      v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (idx < total && r < rows) {
        const T* p = src + (size_t)r * stride + c;
        if (vec && c + 4 <= width) {
          float f[4];
          Quad<T>::load(p, f);
          v[u] = make_float4(f[0], f[1], f[2], f[3]);
        } else {
          if (c < width) v[u].x = to_float(p[0]);
          if (c + 1 < width) v[u].y = to_float(p[1]);
          if (c + 2 < width) v[u].z = to_float(p[2]);
          if (c + 3 < width) v[u].w = to_float(p[3]);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < SC_LOADS; ++u) {
      const int idx = base + u * threads, r = idx / quads, c = (idx - r * quads) * 4;
      if (idx < total) *reinterpret_cast<float4*>(dst + r * ld + c) = v[u];
    }
  }
}

// Whether four neighbouring elements of any row lie in one access (16 bytes of float, 8 of bf16).
template <typename T>
__device__ __forceinline__ bool rows_aligned(const T* p, int stride) { return ((uintptr_t)p & (4 * sizeof(T) - 1)) == 0 && (stride & 3) == 0; }

// Token rows transposed, times `scale`: tile [n][SC_LD] with the token as fast index, zero past the chunk's end and past N.
template <typename T>
__device__ __forceinline__ void load_transposed(const T* src, int stride, int nt, int N, int NP, float* dst, int warp, int warps, int lane,
                                                float scale = 1.f) {
  const bool vec = rows_aligned(src, stride);
  const int t_local = lane & 7, n4 = (lane >> 3) * 4;      // a warp takes 8 tokens x 16 columns
  const int tiles = (SC_Q / 8) * (NP / 16);
  for (int base = warp; base < tiles; base += warps * SC_LOADS) {
    float v[SC_LOADS][4];
#pragma unroll
    for (int u = 0; u < SC_LOADS; ++u) {
      const int tile = base + u * warps, t = (tile & 7) * 8 + t_local, n = (tile >> 3) * 16 + n4;
#pragma unroll
      for (int e = 0; e < 4; ++e) v[u][e] = 0.f;
      if (tile < tiles && t < nt) {
        const T* p = src + (size_t)t * stride + n;
        if (vec && n + 4 <= N) {
          Quad<T>::load(p, v[u]);
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (n + e < N) v[u][e] = to_float(p[e]);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < SC_LOADS; ++u) {
      const int tile = base + u * warps, t = (tile & 7) * 8 + t_local, n = (tile >> 3) * 16 + n4;
      if (tile < tiles) {
#pragma unroll
        for (int e = 0; e < 4; ++e) dst[(n + e) * SC_LD + t] = v[u][e] * scale;
      }
    }
  }
}

}  // namespace ts
