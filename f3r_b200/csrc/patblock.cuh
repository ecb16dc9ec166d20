// patblock.cuh -- the K-column product from row patterns (pattern.cuh).
//
// A tile is one block of 256 rows that share a pattern, a lane a row with K
// accumulators; the windows of x hold K interleaved columns a row, so an entry
// takes one or more 16-byte shared-memory loads, conflict-free from lane to lane,
// where the streamed kernel gathers K values through L1 for every entry (its
// bound: L1 91% busy).  Rows off their block's pattern gather as before.  Same
// multiply-adds in the same order.
// 8 columns, 81^3 27-point stencil, 32-row slices, us a product, streamed -> here:
// fp16 35.2 -> 14.9, Richardson step 37.9 -> 20.4, fp32 47.8 -> 35.3; the solve of 7
// right-hand sides 20.9 -> 15.7 ms.
#pragma once

#include "block.cuh"
#include "pattern.cuh"

namespace f3r {

template <typename V, typename X, typename Epi, int K>
__global__ void __launch_bounds__((kPatWarps + 1) * 32, K * sizeof(typename acc_of<V>::type) <= 32 ? 3 : 2)
    k_pattern_block(PatArgs A, const PatRun<V> *__restrict__ tab, const V *__restrict__ ival, const X *__restrict__ x,
                    Epi epi, int *err) {
  static_assert(kPatBlock == kPatWarps * 32, "a lane a row of a pattern's block");
  epi_setup(epi, 0);
  using Acc = typename acc_of<V>::type;
  constexpr bool H2 = std::is_same<V, __half>::value && std::is_same<X, __half>::value;
  using XB = typename std::conditional<H2, __half, Acc>::type;
  constexpr int RB = K * (int)sizeof(X), PER = RB >= 16 ? 1 : 16 / RB;  // bytes a row, rows a 16-byte unit
  extern __shared__ __align__(128) unsigned char psm[];
  X *stage = reinterpret_cast<X *>(psm);
  PatRun<V> *pats = reinterpret_cast<PatRun<V> *>(psm + (size_t)A.stages * A.elems * RB);
  __shared__ uint64_t full[kPatStages], empty[kPatStages];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t nfl = (int64_t)A.ncols / PER * PER;
  if (threadIdx.x == 0) {
    for (int s = 0; s < A.stages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kPatWarps);
    }
    fence_mbar_init();
  }
  for (int k = threadIdx.x; k < A.np * A.stride; k += blockDim.x) pats[k] = tab[k];
  __syncthreads();
  if (warp == kPatWarps) {  // brings the windows, as in k_sell_pattern
    if (lane != 0) return;
    int i = 0;
    for (int t = blockIdx.x; t < A.ntiles; t += gridDim.x, i++) {
      const int st = i % A.stages;
      if (i >= A.stages && !mbar_wait_bounded(&empty[st], (uint32_t)(i / A.stages - 1) & 1u)) {
        atomicExch(err, (int)DEV_TIMEOUT_SPMV);
        break;
      }
      const int64_t r0 = (int64_t)t * A.tile;
      uint32_t total = 0;
      for (int w = 0; w < A.nwin; w++) {
        const int64_t a = max(r0 + A.win[w].lo, (int64_t)0), b = min(r0 + A.win[w].lo + A.win[w].len, nfl);
        if (a < b) total += (uint32_t)(b - a) * (uint32_t)RB;
      }
      fence_proxy_async_smem();
      mbar_arrive_expect_tx(&full[st], total);
      for (int w = 0; w < A.nwin; w++) {
        const int64_t a = max(r0 + A.win[w].lo, (int64_t)0), b = min(r0 + A.win[w].lo + A.win[w].len, nfl);
        if (a < b)
          bulk_g2s(stage + ((size_t)st * A.elems + A.win[w].base + (a - r0 - A.win[w].lo)) * K, x + a * K,
                   (uint32_t)(b - a) * (uint32_t)RB, &full[st]);
      }
    }
    for (int k = max(0, i - A.stages); k < i; k++) mbar_wait_bounded(&full[k % A.stages], (uint32_t)(k / A.stages) & 1u);
    return;
  }
  for (int q = A.rest.begin(blockIdx.x, gridDim.x); q < A.rest.rounds; q = A.rest.next(q, blockIdx.x, gridDim.x)) {
    const int g = q * kPatWarps + warp;
    if (g >= A.ngroups) break;
    const int32_t r = A.irow[(size_t)g * 32 + lane], k0 = A.iptr[g], w = A.iptr[g + 1] - k0;
    if (r < 0) continue;
    const int32_t *lc = A.icol + (size_t)k0 * 32 + lane;
    const V *lv = ival + (size_t)k0 * 32 + lane;
    Acc acc[K];
#pragma unroll
    for (int c = 0; c < K; c++) acc[c] = 0;
#pragma unroll 2
    for (int k = 0; k < w; k++) {
      XB xg[K];
      RowK<X, K>::ldg(x + (size_t)__ldg(lc + k * 32) * K, xg);
      const V v = __ldg(lv + k * 32);
#pragma unroll
      for (int c = 0; c < K; c++) acc[c] = fma_vx<Acc>(v, xg[c], acc[c]);
    }
    epi.row(r, acc);
  }
  __syncwarp();
  const int q = warp * 32 + lane;  // row in its block
  int st = 0;
  uint32_t phase = 0;
  for (int t = blockIdx.x; t < A.ntiles; t += gridDim.x) {
    const int64_t r0 = (int64_t)t * A.tile;
    const int pid = A.blk[t];
    const bool live = (A.live[(size_t)t * 32 + q % 128 / 4] >> (q / 128 * 4 + q % 4)) & 1;
    X *sx = stage + (size_t)st * A.elems * K;
    if (!mbar_wait_bounded(&full[st], phase)) {
      if (lane == 0) atomicExch(err, (int)DEV_TIMEOUT_SPMV);
      break;
    }
    if (PER > 1 && t >= A.tail_tile) {  // x's last rows, short of a 16-byte unit
      for (int w = 0; w < A.nwin; w++) {
        const int64_t a = r0 + A.win[w].lo, i = nfl + lane;
        if (i < A.ncols && i >= a && i < a + A.win[w].len) {
#pragma unroll
          for (int c = 0; c < K; c++) sx[(A.win[w].base + (i - a)) * K + c] = x[i * K + c];
        }
      }
      __syncwarp();
    }
    Acc acc[K];
#pragma unroll
    for (int c = 0; c < K; c++) acc[c] = 0;
    const PatRun<V> *pr = pats + (size_t)pid * A.stride;
    const int head = pr->at, nr = head & 0xff;
    auto entry = [&](const X *p, V v) {
      XB xg[K];
      RowK<X, K>::load_any(p, xg);
#pragma unroll
      for (int c = 0; c < K; c++) acc[c] = fma_vx<Acc>(v, xg[c], acc[c]);
    };
    for (int k = 1; k <= nr; k++) {
      const PatRun<V> d = pr[k];
      const X *p = sx + (size_t)(q + (d.at & (kPatLong - 1))) * K;
      entry(p, d.v[0]);
      if (d.at >= kPatLong) {
        entry(p + K, d.v[1]);
        entry(p + 2 * K, d.v[2]);
      }
    }
    if (head & kPatPadded) {  // the padding entries: a zero times the row's last x
      const int32_t last = pr[nr].at;
      entry(sx + (size_t)(q + (last & (kPatLong - 1)) + (last >= kPatLong ? 2 : 0)) * K, V(0.0f));
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[st]);
    if (live) epi.row(r0 + q, acc);
    if (++st == A.stages) {
      st = 0;
      phase ^= 1u;
    }
  }
}

}  // namespace f3r
