// pattern.cuh -- products with matrices whose rows repeat: constant-coefficient
// stencils in offset-aligned SELL.
//
// A row's stored entries, as (column - row, value) pairs with the slice's
// padding included, are its pattern.  Where a few patterns cover most rows
// (set-up finds out from the values, make_pattern), the product need not
// stream the matrix: a pattern's offsets and values sit in shared memory, every
// block of 256 rows names one, and the rows that differ from their block's
// pattern (the grid's edges) are kept with their entries, as short lists.  What
// is left to move is x and the result, 42 MB instead of 490 MB for the fp16
// product at 192^3, so the bound shifts to the multiply-adds and to shared
// memory:
//  * x is staged: the offsets are merged into a few windows (three planes of a
//    27-point stencil), and a tile of T rows brings each window into shared
//    memory with one bulk copy, the next tile's while this one is worked;
//  * a lane works 4 consecutive rows: a run of 3 consecutive offsets needs 6
//    values of x, two or three vector loads, for its 12 multiply-adds, where a
//    gather per entry takes 12 loads;
//  * a run's description (where it starts, its values) is one broadcast load
//    for the 256 rows of a warp.
// Every row's multiply-adds are the stored layout's, in its order, padding
// included (a zero times the last x, which only a non-finite x can see), so the
// sums are the streamed kernels' bit for bit.
// What bounds it now is issue (397 warp instructions for 128 rows of 27 entries,
// 108 of them multiply-adds, the other rows' lists included) and, below about a
// million rows, 5 us of set-up and first-tile latency.  27-point stencil, us a product,
// streamed (64-row slices) -> here:  fp16 x fp16  81^3 9.1 -> 5.9, 128^3 28.9 -> 14.4, 192^3
// 86.5 -> 33.5;  fp32  128^3 40.7 -> 18.5, 192^3 130 -> 42;  fp64  128^3 75.0 -> 32.8, 192^3
// 267 -> 100.7.  The 192^3 solve took 93.3 ms with streamed products and 44.3 with these
// and the kernels of blas1.cuh.
// Setting the patterns up reads every row twice on the host: 0.28 s of the 3 s that a
// 192^3 matrix takes to lay out.
#pragma once

#include <algorithm>
#include <vector>

#include "patrest.hpp"
#include "sell.cuh"

namespace f3r {

constexpr int kPatBlock = 256;    // rows that share a pattern: 4 a lane in either half
constexpr int kPatWarps = 8;      // most warps a CTA works rows with (one more brings the windows)
constexpr int kPatStages = 4;     // most tiles in shared memory
constexpr int kPatWindows = 8;    // windows of x
constexpr int kPatRuns = 16;      // runs of a pattern
constexpr int kPatMax = 32;       // patterns of a matrix
constexpr int kPatUnit = 8;       // windows start and end on multiples of 8 elements (16 bytes of fp16)
constexpr int32_t kPatLong = 1 << 24, kPatPadded = 1 << 8, kPatAllLong = 1 << 9;

// A run of 1 or 3 (kPatLong set in at) consecutive offsets: where row 0 of a
// tile finds its first x in the stage, and the values.  The record before a
// pattern's runs holds their number and kPatPadded, kPatAllLong.
template <typename V> struct alignas(16) PatRun {
  int32_t at;
  V v[3];
};

struct PatWindow {
  int32_t lo, len, base;  // first offset (a multiple of 8), elements a tile, first element in the stage
};

struct PatArgs {
  int32_t n, nblk, ntiles, tile;         // rows, 256-row blocks, tiles, rows a tile
  int32_t ncols;                         // columns: the elements of x, what copies and columns stay below
  int32_t np, stride, nwin, elems;       // patterns, records a pattern, windows, elements of a stage
  int32_t stages, tail_tile;             // tiles from tail_tile on reach x's last, partial 16-byte unit
  PatWindow win[kPatWindows];
  const uint8_t *blk;                    // per block: its pattern
  const uint8_t *live;                   // per block and lane: which of its 8 rows follow it (4 of each half)
  int32_t ngroups;                       // the other rows, 32 a group
  PatRest rest;                          // who works them
  const int32_t *irow, *iptr, *icol;     // row (-1: none); first entry / 32 (ngroups + 1); columns, entry k of lane l at k * 32 + l
};

// 4 consecutive values from a 4-element boundary of shared memory
template <typename X> struct Quad;
template <> struct Quad<__half> {
  static __device__ __forceinline__ void ld(const __half *p, __half *o) {
    __half t[4];
    Vec4Load<__half>::ld(p, t);
#pragma unroll
    for (int e = 0; e < 4; e++) o[e] = t[e];
  }
};
template <> struct Quad<float> {
  static __device__ __forceinline__ void ld(const float *p, float *o) {
    const float4 t = *reinterpret_cast<const float4 *>(p);
    o[0] = t.x; o[1] = t.y; o[2] = t.z; o[3] = t.w;
  }
};
template <> struct Quad<double> {
  static __device__ __forceinline__ void ld(const double *p, double *o) {
    const double2 a = *reinterpret_cast<const double2 *>(p), b = *reinterpret_cast<const double2 *>(p + 2);
    o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
  }
};

// One run of 1 or 3 (LNG) offsets for a lane's 4 rows in either half of its
// block: row i takes the values of x from element i of p = row + at on, the
// other half's lie 128 further.
// fp32 and fp64 x: the quads p lies in, M elements into the first.
template <int M, bool LNG, typename X, typename PV, typename Acc>
__device__ __forceinline__ void pat_quads(const X *q, const PV (&v)[3], Acc (&acc)[8]) {
  constexpr int NQ = (M + (LNG ? 6 : 4) + 3) / 4;
#pragma unroll
  for (int h = 0; h < 2; h++) {
    X e[4 * NQ];
#pragma unroll
    for (int k = 0; k < NQ; k++) Quad<X>::ld(q + 128 * h + 4 * k, e + 4 * k);
#pragma unroll
    for (int j = 0; j < (LNG ? 3 : 1); j++)
#pragma unroll
      for (int i = 0; i < 4; i++)
        acc[4 * h + i] = fmaT(to_acc<Acc>(v[j]), to_acc<Acc>(e[M + i + j]), acc[4 * h + i]);
  }
}
template <bool LNG, typename X, typename PV, typename Acc>
__device__ __forceinline__ void pat_run(const X *row, int32_t at, const PV (&v)[3], Acc (&acc)[8]) {
  const X *q = row + (at & ~3);
  switch (at & 3) {
    case 0: pat_quads<0, LNG>(q, v, acc); break;
    case 1: pat_quads<1, LNG>(q, v, acc); break;
    case 2: pat_quads<2, LNG>(q, v, acc); break;
    default: pat_quads<3, LNG>(q, v, acc); break;
  }
}
// fp16 x: the words from the even element at or before p on
template <int M, bool LNG>
__device__ __forceinline__ void pat_words(const uint32_t *q, const __half (&v)[3], float (&acc)[8]) {
  constexpr int NW = (M + (LNG ? 6 : 4) + 1) / 2;
#pragma unroll
  for (int h = 0; h < 2; h++) {
    __half e[2 * NW];
#pragma unroll
    for (int k = 0; k < NW; k++) {
      const uint32_t u = q[64 * h + k];
      const __half2 f = *reinterpret_cast<const __half2 *>(&u);
      e[2 * k] = __low2half(f);
      e[2 * k + 1] = __high2half(f);
    }
#pragma unroll
    for (int j = 0; j < (LNG ? 3 : 1); j++)
#pragma unroll
      for (int i = 0; i < 4; i++) acc[4 * h + i] = fma_vx<float>(v[j], e[M + i + j], acc[4 * h + i]);
  }
}
template <bool LNG>
__device__ __forceinline__ void pat_run(const __half *row, int32_t at, const __half (&v)[3], float (&acc)[8]) {
  const uint32_t *q = reinterpret_cast<const uint32_t *>(row + (at & ~1));
  if (at & 1) pat_words<1, LNG>(q, v, acc);
  else pat_words<0, LNG>(q, v, acc);
}

// epilogues that offer 4 rows at a time (load4 / row4, usable where vec4() holds for the launch's pointers)
template <typename E, typename = void> struct EpiVec4 {
  static constexpr bool has = false;
};
template <typename E> struct EpiVec4<E, decltype((void)&E::vec4)> {
  static constexpr bool has = true;
};
template <typename E> inline bool epi_vec4(const E &e) {
  if constexpr (EpiVec4<E>::has) return e.vec4();
  else return false;
}

// blockDim.x = (warps + 1) * 32: `warps` warps work a tile of warps * kPatBlock
// rows, each its block, and never wait for one another; the last warp's first
// lane keeps the windows of the next tiles coming (a full and an empty mbarrier
// a stage, every wait bounded).
template <typename V, typename X, typename Epi>
__global__ void __launch_bounds__((kPatWarps + 1) * 32, sizeof(V) == 8 ? 2 : 4)
    k_sell_pattern(PatArgs A, const PatRun<V> *__restrict__ tab, const V *__restrict__ ival, const X *x,
                   Epi epi, int vec, int *err) {
  stream_order();
  epi_setup(epi, 0);
  using Acc = typename acc_of<V>::type;
  using XB = typename std::conditional<std::is_same<V, __half>::value && std::is_same<X, __half>::value, __half,
                                       Acc>::type;
  extern __shared__ __align__(128) unsigned char psm[];
  X *stage = reinterpret_cast<X *>(psm);
  PatRun<V> *pats = reinterpret_cast<PatRun<V> *>(psm + (size_t)A.stages * A.elems * sizeof(X));
  __shared__ uint64_t full[kPatStages], empty[kPatStages];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = (blockDim.x >> 5) - 1;
  const int64_t nfl = (int64_t)A.ncols / (16 / (int)sizeof(X)) * (16 / (int)sizeof(X));  // what bulk copies can bring
  if (threadIdx.x == 0) {
    for (int s = 0; s < A.stages; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], warps);
    }
    fence_mbar_init();
  }
  for (int k = threadIdx.x; k < A.np * A.stride; k += blockDim.x) pats[k] = tab[k];
  __syncthreads();
  if (warp == warps) {
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
        if (a < b) total += (uint32_t)(b - a) * (uint32_t)sizeof(X);
      }
      fence_proxy_async_smem();
      mbar_arrive_expect_tx(&full[st], total);
      for (int w = 0; w < A.nwin; w++) {
        const int64_t a = max(r0 + A.win[w].lo, (int64_t)0), b = min(r0 + A.win[w].lo + A.win[w].len, nfl);
        if (a < b)
          bulk_g2s(stage + (size_t)st * A.elems + A.win[w].base + (a - r0 - A.win[w].lo), x + a,
                   (uint32_t)(b - a) * (uint32_t)sizeof(X), &full[st]);
      }
    }
    // the copies in flight land before this thread, and with it the CTA, ends
    for (int k = max(0, i - A.stages); k < i; k++) mbar_wait_bounded(&full[k % A.stages], (uint32_t)(k / A.stages) & 1u);
    return;
  }
  typename Epi::Red none[1];
  // the rows off their block's pattern, while the first windows arrive
  for (int q = A.rest.begin(blockIdx.x, gridDim.x); q < A.rest.rounds; q = A.rest.next(q, blockIdx.x, gridDim.x)) {
    const int g = q * warps + warp;
    if (g >= A.ngroups) break;
    const int32_t r = A.irow[(size_t)g * 32 + lane], k0 = A.iptr[g], w = A.iptr[g + 1] - k0;
    if (r < 0) continue;
    const int32_t *lc = A.icol + (size_t)k0 * 32 + lane;
    const V *lv = ival + (size_t)k0 * 32 + lane;
    const typename Epi::Pre pre = epi.load(r);
    Acc acc = 0;
    // 4 entries at a time (widths are multiples of 4), the next ones' columns and values ahead of the gathers
    int32_t c[4];
    V v[4];
    auto entries = [&](int k) {
#pragma unroll
      for (int e = 0; e < 4; e++) {
        c[e] = __ldg(lc + (k + e) * 32);
        v[e] = __ldg(lv + (k + e) * 32);
      }
    };
    if (w > 0) entries(0);
    for (int k = 0; k < w; k += 4) {
      XB xg[4];
      V u[4];
#pragma unroll
      for (int e = 0; e < 4; e++) {
        xg[e] = to_acc<XB>(ld_stream(x + c[e]));
        u[e] = v[e];
      }
      if (k + 4 < w) entries(k + 4);
#pragma unroll
      for (int e = 0; e < 4; e++) acc = fma_vx<Acc>(u[e], xg[e], acc);
    }
    epi.row(r, acc, pre, none);
  }
  __syncwarp();
  int64_t b = (int64_t)blockIdx.x * warps + warp;
  const int64_t step = (int64_t)gridDim.x * warps;
  int pid = b < A.nblk ? A.blk[b] : 0;
  uint32_t live = b < A.nblk ? A.live[b * 32 + lane] : 0;
  int st = 0;
  uint32_t phase = 0;
  for (int t = blockIdx.x; t < A.ntiles; t += gridDim.x, b += step) {
    const int64_t r0 = (int64_t)t * A.tile, r = b * kPatBlock + 4 * lane;
    X *sx = stage + (size_t)st * A.elems;
    // the next block's pattern and rows, ahead of its tile
    const int npid = b + step < A.nblk ? A.blk[b + step] : 0;
    const uint32_t nlive = b + step < A.nblk ? A.live[(b + step) * 32 + lane] : 0;
    // the epilogue's operands, ahead of the sums
    typename Epi::Pre pre[8];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int64_t q = r + 128 * h;
      typename Epi::Pre t4[4];
      bool four = false;
      if constexpr (EpiVec4<Epi>::has) {
        four = vec && q + 3 < A.n;
        if (four) epi.load4(q, t4);
      }
      if (!four) {
#pragma unroll
        for (int i = 0; i < 4; i++)
          if ((live >> (4 * h + i)) & 1u) t4[i] = epi.load(q + i);
      }
#pragma unroll
      for (int i = 0; i < 4; i++) pre[4 * h + i] = t4[i];
    }
    if (!mbar_wait_bounded(&full[st], phase)) {
      if (lane == 0) atomicExch(err, (int)DEV_TIMEOUT_SPMV);
      break;
    }
    if (t >= A.tail_tile) {
      // x's last elements, short of a 16-byte unit: every warp that may read them writes them (the same values)
      for (int w = 0; w < A.nwin; w++) {
        const int64_t a = r0 + A.win[w].lo, i = nfl + lane;
        if (i < A.ncols && i >= a && i < a + A.win[w].len) sx[A.win[w].base + (i - a)] = x[i];
      }
      __syncwarp();
    }
    Acc acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    const PatRun<V> *pr = pats + (size_t)pid * A.stride;
    const int head = pr->at, nr = head & 0xff;
    const X *row = sx + (r - r0);
    if (head & kPatAllLong) {
      for (int k = 1; k <= nr; k++) {
        const PatRun<V> d = pr[k];
        pat_run<true>(row, d.at & (kPatLong - 1), d.v, acc);
      }
    } else {
      for (int k = 1; k <= nr; k++) {
        const PatRun<V> d = pr[k];
        if (d.at >= kPatLong) pat_run<true>(row, d.at & (kPatLong - 1), d.v, acc);
        else pat_run<false>(row, d.at, d.v, acc);
      }
    }
    if (head & kPatPadded) {  // the padding entries: a zero times the row's last x
      const int32_t last = pr[nr].at;
      const X *q = row + (last & (kPatLong - 1)) + (last >= kPatLong ? 2 : 0);
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int i = 0; i < 4; i++) acc[4 * h + i] = fmaT(Acc(0), to_acc<Acc>(q[128 * h + i]), acc[4 * h + i]);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[st]);
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int64_t q = r + 128 * h;
      const uint32_t rows = (live >> (4 * h)) & 15u;
      Acc a4[4];
      typename Epi::Pre t4[4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        a4[i] = acc[4 * h + i];
        t4[i] = pre[4 * h + i];
      }
      bool four = false;
      if constexpr (EpiVec4<Epi>::has) {
        four = vec && q + 3 < A.n;
        if (four) epi.row4(q, a4, t4, rows);
      }
      if (!four) {
#pragma unroll
        for (int i = 0; i < 4; i++)
          if ((rows >> i) & 1u) epi.row(q + i, a4[i], t4[i], none);
      }
    }
    pid = npid;
    live = nlive;
    if (++st == A.stages) {
      st = 0;
      phase ^= 1u;
    }
  }
}

// A matrix's patterns on the device (DeviceSell::pat)
struct DevPattern {
  PatArgs a{};
  int warps = 0;
  PatArgs ab{};  // for tiles of one block (patblock.cuh); ntiles = 0: too many windows
  int32_t listed_rows = 0;     // off their block's pattern
  int64_t listed_entries = 0;  // of their lists, padding included
  // the patterns' records, for a's tiles and for ab's
  PatRun<double> *t64[2] = {nullptr, nullptr};
  PatRun<float> *t32[2] = {nullptr, nullptr};
  PatRun<__half> *t16[2] = {nullptr, nullptr};
  double *v64 = nullptr;
  float *v32 = nullptr;
  __half *v16 = nullptr;
  std::vector<void *> allocs;
  // what a product reads of the matrix, with values of sv bytes
  int64_t bytes(size_t sv) const {
    return listed_entries * (int64_t)(sv + 4) + a.ngroups * (int64_t)(32 * 4 + 4) + a.nblk * (int64_t)33;
  }
  const PatRun<double> *tab(const double *, int i = 0) const { return t64[i]; }
  const PatRun<float> *tab(const float *, int i = 0) const { return t32[i]; }
  const PatRun<__half> *tab(const __half *, int i = 0) const { return t16[i]; }
  const double *vals(const double *) const { return v64; }
  const float *vals(const float *) const { return v32; }
  const __half *vals(const __half *) const { return v16; }
  ~DevPattern() {
    for (void *p : allocs) cudaFree(p);
  }
};

// CTAs an SM and stages of x for elements of sx bytes and table records of st
// bytes: the most CTAs that leave two stages or more each
struct PatShape {
  int stages = 0, ctas = 0;
  size_t smem = 0;
};
// Rows from which the patterns pay: one wave of the streamed kernel's rows where
// that kernel is at its best (fp16 values, 64-row slices: 64^3 5.5 us streamed,
// 6.1 here, 81^3 9.1 and 5.9), half of that elsewhere (32-row slices at 64^3: 7.5
// and 6.1; fp32 8.4 and 6.6, fp64 12.4 and 7.9; at 48^3 no gain is left).
inline int64_t pattern_rows(int sm_count, int height, size_t sv) {
  return (int64_t)sm_count * (height == 64 && sv == 2 ? 2048 : 1024);
}
// the first tile whose windows pass the last of x that whole units of `per` elements bring
inline int32_t pattern_tail(const PatArgs &a, int64_t per) {
  int64_t hi = 0;
  for (int w = 0; w < a.nwin; w++) hi = std::max<int64_t>(hi, (int64_t)a.win[w].lo + a.win[w].len);
  const int64_t nfl = a.ncols / per * per;
  return nfl == a.ncols ? a.ntiles : (int32_t)std::max<int64_t>(0, (nfl - hi) / a.tile);
}
inline PatShape pattern_shape(const PatArgs &a, int warps, size_t sx, size_t st) {
  const size_t one = (size_t)a.elems * sx, table = (size_t)a.np * a.stride * st, sm = 227 * 1024;
  for (int ctas = 32 / warps; ctas >= 1; ctas--) {
    const size_t room = sm / ctas - 1024 - 256;
    for (int stages = kPatStages; stages >= 2; stages--)
      if (stages * one + table <= room) return PatShape{stages, ctas, stages * one + table};
  }
  return PatShape();
}

}  // namespace f3r
