// direct.cuh -- SELL products with a thread a row and plain loads.
//
// The bulk-copy kernels (sell.cuh) stream slices of many columns through
// shared memory; a copy, an mbarrier round trip and a slice's metadata are then
// spread over thousands of bytes.  Two kinds of matrices do not pay for that
// and come here (launch_sell's rule):
//  * short rows (at most kDirectShort stored columns: 7-point matrices, SDAINV
//    factors), where a 32-row slice of 4 columns is a 256-byte copy;
//  * small matrices with packed rows, whose rows are all resident at once: the bulk kernel's time is then one warp's chain of waits.
// Every thread issues the loads of its row before it uses any of them (in an
// offset-aligned slice the row's values are contiguous, 8 to 64 bytes), and the
// SM holds 40 to 64 warps of them.  What bounds it is the latency of the two
// dependent steps (slot bases or columns, then x) times the waves of rows; two
// rows a lane (R = 2) halve the waves where there are several.  Sums are formed in stored
// order with the same multiply-adds over the same entries (padding included),
// so the results are the bulk kernels' bit for bit.
//
// fp16 values and x, us a product, bulk kernel -> this one:
//   7-point aligned, 64-row slices:  64^3 3.6 -> 2.5, 128^3 15.0 -> 9.4, 200^3 50.8 -> 33.2 (180 MB: 5.4 TB/s)
//   7-point aligned, 32-row slices:  64^3 4.9 -> 2.5, 128^3 23.7 -> 10.4, 200^3 84.0 -> 38.5
//   7-point packed:                  64^3 6.3 -> 3.7, 100^3 15.2 -> 8.7, 128^3 29.5 -> 26.5
//   27-point packed:                 16^3 4.0 -> 3.1, 64^3 10.8 -> 7.1 (80^3: 16.9 -> 16.4, left to the bulk kernel)
#pragma once

#include "sell.cuh"

namespace f3r {

constexpr int kDirectThreads = 256;
constexpr int kDirectShort = 8;       // widest row of the short form
constexpr int kDirectResident = 2048;  // rows of a small matrix per SM: one wave of threads
// Values and columns of a small matrix: sv bytes an entry and 4 for its column.
// Plain loads pay off while the matrix stays in the 126 MB L2 beside x from one
// product to the next; the bulk kernel streams past it.  Short fp32 rows (more than
// half a wave of them) may take a little more.  Bulk kernel -> thread a row, us a
// product: 150,000 x 80 fp16 (72 MB) 16.5 -> 14.4, 20,000 x 500 fp32 (80 MB) 43 -> 27,
// 160,000 x 90 fp16 (86 MB) 20.6 -> 22.6, 110,000 x 140 fp16 (92 MB) 17.6 -> 24.5, 20,000 x
// 1,000 fp16 (120 MB) 71 -> 131; 300,000 x 40 fp32 (96 MB) 20.4 -> 16.5, x 56 (134 MB) 26.0
// -> 28.4, x 64 fp16 (115 MB) 22.4 -> 28.7.
inline bool direct_bytes_fit(int64_t entries, size_t sv, int64_t n, int64_t wave) {
  return entries * (int64_t)(sv + 4) <= (sv == 4 && n * 2 > wave ? 97000000 : 80000000);
}

// N consecutive values (4 or 8, from a multiple of N) in accesses of up to 32 bytes, not kept in L1
template <typename V, int N> __device__ __forceinline__ void ld_row(const V *p, V (&o)[N]) {
  constexpr int B = (int)sizeof(V) * N;
  if constexpr (B % 32 == 0) {
#pragma unroll
    for (int q = 0; q < B / 32; q++) {
      uint32_t u[8];
      asm volatile("ld.global.nc.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                   : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
                   : "l"(reinterpret_cast<const char *>(p) + 32 * q));
      const V *t = reinterpret_cast<const V *>(u);
#pragma unroll
      for (int e = 0; e < 32 / (int)sizeof(V); e++) o[q * (32 / (int)sizeof(V)) + e] = t[e];
    }
  } else if constexpr (B == 16) {
    uint32_t u[4];
    asm volatile("ld.global.nc.L1::no_allocate.v4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3])
                 : "l"(p));
    const V *t = reinterpret_cast<const V *>(u);
#pragma unroll
    for (int e = 0; e < N; e++) o[e] = t[e];
  } else {
    static_assert(B == 8, "row access");
    uint32_t u[2];
    asm volatile("ld.global.nc.L1::no_allocate.v2.b32 {%0,%1}, [%2];" : "=r"(u[0]), "=r"(u[1]) : "l"(p));
    const V *t = reinterpret_cast<const V *>(u);
#pragma unroll
    for (int e = 0; e < N; e++) o[e] = t[e];
  }
}

// R rows of one lane, rows r0 + 32 i (i < R; r0 + 32 i < n where bit i of live
// is set), of offset-aligned slices W slots wide at most: W = 4 or 8
template <int W, int R, int H, typename V, typename X, typename Acc>
__device__ __forceinline__ void direct_aligned_rows(const V *val, const DevSell &A, const X *x, int64_t r0,
                                                    Acc (&acc)[R]) {
  using XB = typename std::conditional<std::is_same<V, __half>::value && std::is_same<X, __half>::value, __half,
                                       Acc>::type;
  constexpr int NS = R * 32 > H ? R * 32 / H : 1;  // slices of the R rows (r0 - lane is a multiple of 32 R)
  V v[R][W];
  XB xg[R][W];
  int32_t b[NS][W];
  int cp[NS];
#pragma unroll
  for (int i = 0; i < R; i++)
    if (r0 + 32 * i < A.n) ld_row<V, W>(val + (size_t)(r0 + 32 * i) * W, v[i]);
#pragma unroll
  for (int k = 0; k < NS; k++) {
    const int32_t s = (int32_t)(r0 / H) + k;
    if (s < A.nslices) {
      cp[k] = A.cbptr[s];
#pragma unroll
      for (int g = 0; g < W / 4; g++) {
        const int4 q = __ldg(reinterpret_cast<const int4 *>(A.cbase + (size_t)s * W) + g);
        b[k][4 * g] = q.x; b[k][4 * g + 1] = q.y; b[k][4 * g + 2] = q.z; b[k][4 * g + 3] = q.w;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < R; i++) {
    const int k = NS > 1 ? i * 32 / H : 0, q = (int)((r0 + 32 * i) % H);
    if (r0 + 32 * i < A.n) {
#pragma unroll
      for (int e = 0; e < W; e++) {
        int32_t c = b[k][e] + q;
        if (cp[k] & 1) c = min(max(c, 0), A.ncols - 1);
        xg[i][e] = to_acc<XB>(ld_stream(x + c));
      }
    }
  }
#pragma unroll
  for (int i = 0; i < R; i++)
#pragma unroll
    for (int e = 0; e < W; e++) acc[i] = fma_vx<Acc>(v[i][e], xg[i][e], acc[i]);
}

// Offset-aligned slices of one width, 4 or 8 slots (A.uw): warp w works rows
// 32 R w ... , R a lane
template <typename V, typename X, typename Epi, int H, int R>
__global__ void __launch_bounds__(kDirectThreads)
    k_sell_direct_aligned(const V *__restrict__ val, DevSell A, const X *x, Epi epi) {
  stream_order();
  epi_setup(epi, 0);
  using Acc = typename acc_of<V>::type;
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, r0 = t / 32 * (32 * R) + t % 32;
  if (r0 >= A.n) return;
  typename Epi::Pre pre[R];
  Acc acc[R];
#pragma unroll
  for (int i = 0; i < R; i++) {
    acc[i] = 0;
    if (r0 + 32 * i < A.n) pre[i] = epi.load(r0 + 32 * i);
  }
  if (A.uw == 8) direct_aligned_rows<8, R, H>(val, A, x, r0, acc);
  else direct_aligned_rows<4, R, H>(val, A, x, r0, acc);
  typename Epi::Red none[1];
#pragma unroll
  for (int i = 0; i < R; i++)
    if (r0 + 32 * i < A.n) epi.row(r0 + 32 * i, acc[i], pre[i], none);
}

// Offset-aligned slices that are not all alike: 4 or 8 slots wide (or empty),
// or with explicit columns among them (the mixed form); a row a lane
template <typename V, typename X, typename Epi, int H>
__global__ void __launch_bounds__(kDirectThreads)
    k_sell_direct_mixed(const V *__restrict__ val, DevSell A, const X *x, Epi epi) {
  stream_order();
  epi_setup(epi, 0);
  using Acc = typename acc_of<V>::type;
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= A.n) return;
  const int32_t s = (int32_t)(r / H), q = (int32_t)(r % H);
  const int32_t s0 = A.sptr[s], w = A.sptr[s + 1] - s0, cp = A.cbptr[s], xo = A.xoff ? A.xoff[s] : -1;
  const typename Epi::Pre pre = epi.load(r);
  const V *lv = val + (size_t)s0 * H + (size_t)q * w;
  Acc acc = 0;
  auto row = [&](auto wc) {
    constexpr int W = decltype(wc)::value;
    using XB = typename std::conditional<std::is_same<V, __half>::value && std::is_same<X, __half>::value, __half,
                                         Acc>::type;
    V v[W];
    XB xg[W];
    int32_t c[W];
    ld_row<V, W>(lv, v);
    if (xo < 0) {
#pragma unroll
      for (int g = 0; g < W / 4; g++) {
        const int4 b = __ldg(reinterpret_cast<const int4 *>(A.cbase + (cp & ~3)) + g);
        c[4 * g] = b.x + q; c[4 * g + 1] = b.y + q; c[4 * g + 2] = b.z + q; c[4 * g + 3] = b.w + q;
      }
      if (!A.xoff && (cp & 1)) {
#pragma unroll
        for (int e = 0; e < W; e++) c[e] = min(max(c[e], 0), A.ncols - 1);
      }
    } else {
#pragma unroll
      for (int e = 0; e < W; e++) c[e] = __ldg(A.col + (size_t)xo + e * 32 + q);
    }
#pragma unroll
    for (int e = 0; e < W; e++) xg[e] = to_acc<XB>(ld_stream(x + c[e]));
#pragma unroll
    for (int e = 0; e < W; e++) acc = fma_vx<Acc>(v[e], xg[e], acc);
  };
  if (w == 8) row(std::integral_constant<int, 8>());
  else if (w == 4) row(std::integral_constant<int, 4>());
  typename Epi::Red none[1];
  epi.row(r, acc, pre, none);
}

// Packed int32 slices, UNR columns at a time
template <typename V, typename X, typename Epi, int UNR>
__global__ void __launch_bounds__(kDirectThreads)
    k_sell_direct_packed(const V *__restrict__ val, DevSell A, const X *x, Epi epi) {
  stream_order();
  epi_setup(epi, 0);
  using Acc = typename acc_of<V>::type;
  using XB = typename std::conditional<std::is_same<V, __half>::value && std::is_same<X, __half>::value, __half,
                                       Acc>::type;
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= A.n) return;
  const int32_t s = (int32_t)(r / 32);
  const int32_t s0 = A.uw > 0 ? s * A.uw : A.sptr[s], w = A.uw > 0 ? A.uw : A.sptr[s + 1] - s0;
  const typename Epi::Pre pre = epi.load(r);
  Acc acc = 0;
  const V *lv = val + (size_t)s0 * 32 + r % 32;
  const int32_t *lc = A.col + (size_t)s0 * 32 + r % 32;
  auto part = [&](int k0, auto full) {
    int32_t c[UNR];
    V v[UNR];
    XB xg[UNR];
#pragma unroll
    for (int e = 0; e < UNR; e++)
      if (full || k0 + e < w) {
        c[e] = __ldg(lc + (k0 + e) * 32);
        v[e] = __ldg(lv + (k0 + e) * 32);
      }
#pragma unroll
    for (int e = 0; e < UNR; e++)
      if (full || k0 + e < w) xg[e] = to_acc<XB>(ld_stream(x + c[e]));
#pragma unroll
    for (int e = 0; e < UNR; e++)
      if (full || k0 + e < w) acc = fma_vx<Acc>(v[e], xg[e], acc);
  };
  int k0 = 0;
  for (; k0 + UNR <= w; k0 += UNR) part(k0, std::true_type());
  if (k0 < w) part(k0, std::false_type());
  typename Epi::Red none[1];
  epi.row(r, acc, pre, none);
}

}  // namespace f3r
