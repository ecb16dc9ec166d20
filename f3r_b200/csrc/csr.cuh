// csr.cuh -- CSR SpMV with the SELL kernel's epilogues (the format = CSR
// option of the solver and F3R_SELL_CSR matrices).  The reference's CSR
// operate is matrix/csr.hpp's; its GPU drivers use SELL<32>.
//
// A warp takes a group of 32 rows, lane l row 32 g + l.  The group's contiguous
// CSR range (in tiles of T entries) is widened to 16-byte boundaries and copied
// to shared memory with 16-byte cp.async, and each lane sums its own row in
// column order, B gathers at a time: the packed SELL layout's sums bit for bit
// (SELL's padding adds exact zeros).  The value and index arrays carry kCsrPad
// elements of padding, so the widened copies stay inside their allocations.
//
// What bounds it is each group's chain of waits (row pointers, copy, one or two
// rounds of gathers), so the more groups an SM holds the better: blocks of 4
// warps that the hardware schedules as others finish, one tile of shared memory a
// warp, and tiles of kCsrShort entries where every group fits them (rows of at
// most 8 entries: 64 warps an SM; 128^3 7-point, fp32: 27.5 us, 52.4 with
// kCsrWide), of kCsrMid where every group fits those (rows of 9 to 16; 10^6 x 10,
// kCsrWide -> kCsrMid: fp32 24.4 -> 18.5 us, fp64 45.3 -> 32.9) and for fp64 rows of
// up to 64, whose wide tiles leave 16 warps an SM (300,000 x 40 61.4 -> 55.3, x 64
// 159.9 -> 152.7; x 100 113.9 -> 148), of kCsrWide otherwise.  Against 24 persistent warps an SM with a
// two-stage ring of 512 entries: 27-point, fp16, 40^3 7.4 -> 4.1 us, 64^3 17.5 ->
// 9.4, 128^3 109 -> 74; 7-point 64^3 6.5 -> 4.4, 200^3 147 -> 100.
#pragma once

#include "sell.cuh"

namespace f3r {

constexpr int kCsrWide = 1024, kCsrMid = 512, kCsrShort = 256;  // entries a tile
constexpr int kCsrWarps = 4;                     // warps a block
constexpr int kCsrPad = 16;                      // elements of padding after the value and index arrays

template <typename V, int T> constexpr uint32_t csr_tile_bytes() { return T * sizeof(V) + 32 + T * 4 + 32; }

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

template <typename V, typename X, typename Epi, int T>
__global__ void __launch_bounds__(kCsrWarps * 32)
    k_csr_group(const V *__restrict__ val, DevSell A, const X *x, Epi epi) {
  stream_order();
  epi_setup(epi, 0);
  using Acc = typename acc_of<V>::type;
  constexpr int B = T == kCsrShort ? 8 : 16;  // gathers in flight per lane
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t g = (int64_t)blockIdx.x * kCsrWarps + warp, r = g * 32 + lane;
  if (g >= A.nslices) return;
  unsigned char *vbuf = smem + (size_t)warp * csr_tile_bytes<V, T>(), *ibuf = vbuf + T * sizeof(V) + 32;
  const bool live = r < A.n;
  const int32_t rb = A.rptr[live ? r : A.n], re = A.rptr[live ? r + 1 : A.n];
  const int32_t gb = __shfl_sync(0xffffffffu, rb, 0), ge = __shfl_sync(0xffffffffu, re, 31);
  typename Epi::Pre pre{};
  if (live) pre = epi.load(r);
  Acc acc = 0;
  for (int32_t t0 = gb; t0 < ge; t0 += T) {
    const int cnt = min(T, ge - t0);
    // the tile's byte ranges widened to 16-byte units (the arrays carry kCsrPad elements)
    const size_t b0 = (size_t)t0 * sizeof(V), a0 = b0 & ~(size_t)15, c0 = (size_t)t0 * 4, d0 = c0 & ~(size_t)15;
    const int nv = (int)((b0 + cnt * sizeof(V) + 15 - a0) / 16), ni = (int)((c0 + (size_t)cnt * 4 + 15 - d0) / 16);
    const char *vs = reinterpret_cast<const char *>(val) + a0, *is = reinterpret_cast<const char *>(A.col) + d0;
    for (int k = lane; k < ni; k += 32) cp_async16(ibuf + k * 16, is + k * 16);
    for (int k = lane; k < nv; k += 32) cp_async16(vbuf + k * 16, vs + k * 16);
    cp_async_commit();
    cp_async_wait<0>();
    __syncwarp();
    const V *sv = reinterpret_cast<const V *>(vbuf + (b0 - a0));
    const int32_t *sc = reinterpret_cast<const int32_t *>(ibuf + (c0 - d0));
    const int lo = max(rb, t0) - t0, hi = min(re, t0 + cnt) - t0;
    for (int k = lo; k < hi; k += B) {
      Acc xv[B];
#pragma unroll
      for (int e = 0; e < B; e++)
        if (k + e < hi) xv[e] = to_acc<Acc>(ld_stream(x + sc[k + e]));
#pragma unroll
      for (int e = 0; e < B; e++)
        if (k + e < hi) acc = fmaT(to_acc<Acc>(sv[k + e]), xv[e], acc);
    }
    __syncwarp();  // every lane is done with the tile before it is refilled
  }
  typename Epi::Red none[1];
  if (live) epi.row(r, acc, pre, none);
}

}  // namespace f3r
