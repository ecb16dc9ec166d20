// blockdots.cuh -- the Gram-Schmidt dot products of the fp32 levels over K
// columns: H(j, k)(c) = <w(:, c), V(k)(:, c)>, k < nv <= 8.
//
// The sums of the single-column k_dots1 (blas1.cuh), column by column: a grid of
// blocks of 256 threads, a thread sums rows 4q .. 4q + 3, q = tid, tid + stride,
// ...; butterflies, the 8 warps in order, the blocks by t = t, t + 256, .... A
// thread's 4 rows are 16 K contiguous bytes, so its own loads would leave the
// lanes of an access 16 K bytes apart; instead a warp moves its contiguous tile
// (32 threads' rows of one vector) with coalesced 16-byte loads, the next
// vector's while the current one is worked, and hands it over through shared
// memory (a padded run a thread, as k_cgs_updateK).  A warp's 8 values are
// reduced together, and so are a thread's 8 of the final stage.
// 8 columns, us a call averaged over a solve (the per-thread loads before -> here):
// 531,441 rows 40.3 -> 21.5, 110,592 rows 13.6 -> 7.3; two blocks an SM (128
// registers) against one: 21.5 and 27.4.
#pragma once

#include "blas1.cuh"

namespace f3r {

constexpr int kDotsPass = 4;  // vectors a pass over w

template <int K> constexpr size_t dots_stage_bytes() { return (size_t)8 * 32 * (4 * K + 4) * sizeof(float); }

template <int K>
__global__ void __launch_bounds__(256, K == 16 ? 1 : 2)
    k_dotsK(const float *__restrict__ w, Cols<float> V, int nv, int64_t n, GridRed gr, float *__restrict__ hcol,
            int64_t hstride) {
  constexpr int NV = kDotsPass, S = 4 * K, P = S + 4;  // values a thread, its padded pitch
  static_assert(K >= 2 && NV * K % 8 == 0, "whole groups of 8 values");
  extern __shared__ __align__(16) float dots_stage[];
  __shared__ float sred[8][NV * K];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float *tile = dots_stage + warp * 32 * P;
  const float *mine = tile + lane * P;
  float *part = static_cast<float *>(gr.partials);
  const int ntot = nv * K;
  const int64_t stride = (int64_t)gridDim.x * 256, nq = n / 4, tid = (int64_t)blockIdx.x * 256 + threadIdx.x;
  for (int k0 = 0; k0 < nv; k0 += NV) {
    const int m = min(NV, nv - k0);
    float a[NV][K];
#pragma unroll
    for (int k = 0; k < NV; k++)
#pragma unroll
      for (int c = 0; c < K; c++) a[k][c] = 0.0f;
    for (int64_t q0 = tid - lane; q0 < nq; q0 += stride) {
      const int lim = (int)((nq - q0 < 32 ? nq - q0 : 32) * S);  // values of the tile inside the vector
      float4 u[K];
      auto fetch = [&](const float *src) {
#pragma unroll
        for (int i = 0; i < K; i++)
          if (lane * 4 + 128 * i < lim) u[i] = __ldg(reinterpret_cast<const float4 *>(src + q0 * S) + lane + 32 * i);
      };
      auto hand_over = [&]() {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < K; i++) {
          const int at = lane * 4 + 128 * i;
          if (at < lim) *reinterpret_cast<float4 *>(tile + at / S * P + at % S) = u[i];
        }
        __syncwarp();
      };
      float x[S];
      fetch(w);
      hand_over();
      fetch(V.p[k0]);
#pragma unroll
      for (int e = 0; e < S; e += 4) {
        const float4 t = *reinterpret_cast<const float4 *>(mine + e);
        x[e] = t.x; x[e + 1] = t.y; x[e + 2] = t.z; x[e + 3] = t.w;
      }
      const bool own = q0 + lane < nq;
#pragma unroll
      for (int k = 0; k < NV; k++)
        if (k < m) {
          hand_over();
          if (k + 1 < m) fetch(V.p[k0 + k + 1]);
          if (own) {
#pragma unroll
            for (int e = 0; e < S; e += 4) {
              const float4 t = *reinterpret_cast<const float4 *>(mine + e);
              a[k][e % K] = __fmaf_rn(x[e], t.x, a[k][e % K]);
              a[k][(e + 1) % K] = __fmaf_rn(x[e + 1], t.y, a[k][(e + 1) % K]);
              a[k][(e + 2) % K] = __fmaf_rn(x[e + 2], t.z, a[k][(e + 2) % K]);
              a[k][(e + 3) % K] = __fmaf_rn(x[e + 3], t.w, a[k][(e + 3) % K]);
            }
          }
        }
    }
    if (tid < n - nq * 4) {  // the last n % 4 rows: the first threads
      const int64_t i = (nq * 4 + tid) * K;
#pragma unroll
      for (int k = 0; k < NV; k++)
        if (k < m) {
#pragma unroll
          for (int c = 0; c < K; c++) a[k][c] = __fmaf_rn(w[i + c], V.p[k0 + k][i + c], a[k][c]);
        }
    }
#pragma unroll
    for (int g = 0; g < NV * K / 8; g++) {
      float v[8];
#pragma unroll
      for (int i = 0; i < 8; i++) v[i] = a[(8 * g + i) / K][(8 * g + i) % K];
      const float t = WarpSums<8>::run(v);
      if (WarpSums<8>::writes(lane)) sred[warp][8 * g + WarpSums<8>::index_of(lane)] = t;
    }
    __syncthreads();
    if ((int)threadIdx.x < m * K) {
      float s = 0.0f;
#pragma unroll
      for (int q = 0; q < 8; q++) s += sred[q][threadIdx.x];
      part[(size_t)blockIdx.x * ntot + k0 * K + threadIdx.x] = s;
    }
    __syncthreads();
  }
  if (!last_block1(gr.ticket)) return;
  __shared__ float sw[8][8];
#pragma unroll 2
  for (int q = 0; q < ntot; q += 8) {
    float s[8];
#pragma unroll
    for (int i = 0; i < 8; i++) s[i] = 0.0f;
#pragma unroll 5
    for (int b = threadIdx.x; b < (int)gridDim.x; b += 256) {
#pragma unroll
      for (int i = 0; i < 8; i++)
        if (q + i < ntot) s[i] += __ldcg(part + (size_t)b * ntot + q + i);
    }
    const float v = WarpSums<8>::run(s);
    if (WarpSums<8>::writes(lane)) sw[warp][WarpSums<8>::index_of(lane)] = v;
    __syncthreads();
    const int t = threadIdx.x;
    if (t < 8 && q + t < ntot) {
      float r = 0.0f;
#pragma unroll
      for (int i = 0; i < 8; i++) r += sw[i][t];
      hcol[((q + t) % K) * hstride + (q + t) / K] = r;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) *gr.ticket = 0;
}

}  // namespace f3r
