// ilu.cuh -- block-Jacobi ILU(0) triangular solves on the GPU.
//
// The reference solves each block sequentially on one CPU thread
// (trsv/bj.hpp:58-98).  Here every block-Jacobi block is one CTA, and inside
// a block the rows are grouped into dependency levels (level(i) = 1 + the
// highest level among the rows it reads); a CTA sweeps its levels in order
// with one __syncthreads() between levels, one thread per row.  The blocks
// never read each other's rows, so no inter-CTA synchronisation exists.
// Arithmetic per row follows the reference's order: the forward sweep walks
// the row's off-diagonals by increasing column, the backward sweep by
// decreasing column (the reference's 180-degree rotated U, csr.hpp:60-86)
// and multiplies by the fp16-rounded inverse diagonal formed in fp64
// (CSR::inverse_last, csr.hpp:60-65).  fp16 values, fp32 accumulation.
#pragma once

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "device.cuh"
#include "internal.hpp"

namespace f3r {

struct RichState;

struct IluTri {
  // the factor laid out in (block, level) row order q, as the kernel visits it
  int4 *meta = nullptr;    // per q: vector position, first and end entry, unused
  __half *val = nullptr;   // entries of every row in processing order (diagonal excluded)
  int32_t *idx = nullptr;  // their columns, mapped to vector positions
  __half *dinv = nullptr;  // upper only: fp16(1 / u_ii), per q
  int32_t *lvl_off = nullptr;  // row ranges (in q) of the levels, all blocks
  int32_t *blk_lvl = nullptr;  // per block: first level index (nblocks + 1)
};

// One CTA per block-Jacobi block, rows level by level; the factor stays in
// global memory.  Used where the blocks' rows do not occupy contiguous vector
// positions (sigma-sorted rows) or a block or row is too large for
// k_bj_stream below.
template <bool UPPER>
__global__ void k_trsv_bj(IluTri T, const __half *__restrict__ in, __half *__restrict__ out,
                          const __half *__restrict__ ome) {
  const int b = blockIdx.x;
  const int l0 = T.blk_lvl[b], l1 = T.blk_lvl[b + 1];
  const float om = ome ? __half2float(*ome) : 1.0f;
  for (int l = l0; l < l1; l++) {
    const int r0 = T.lvl_off[l], r1 = T.lvl_off[l + 1];
    for (int q = r0 + threadIdx.x; q < r1; q += blockDim.x) {
      const int4 m = T.meta[q];
      float t = __half2float(in[m.x]);
      for (int32_t j = m.y; j < m.z; j++)
        t = __fmaf_rn(-__half2float(T.val[j]), __half2float(out[T.idx[j]]), t);
      out[m.x] = UPPER ? __float2half_rn(t * __half2float(T.dinv[q])) : __float2half_rn(t);
    }
    __syncthreads();
  }
  // the reference solves, then scales: hout *= ome[0] (work/src/f3r.cpp:216, 229)
  if (UPPER && ome) {
    for (int q = T.lvl_off[l0] + threadIdx.x; q < T.lvl_off[l1]; q += blockDim.x) {
      const int32_t p = T.meta[q].x;
      out[p] = __float2half_rn(__half2float(out[p]) * om);
    }
  }
}

// ---------------------------------------------------------------------------
// Both triangular solves of a block in one CTA, the block's vector in shared
// memory and its factors streamed through a ring of bulk copies.
//
// The time of a block solve is its chain of dependency levels (137 levels of
// 17 rows for a 64^3 27-point matrix over 112 blocks), so what counts is the
// latency of one level.  Each factor is packed, in the order the kernel visits
// rows, into chunks of kBjChunk bytes: the row ranges that may run in parallel
// ("parts", a level or a piece of one), 4 bytes a row (position in the block,
// fp16 inverse diagonal) and 4 bytes an entry (fp16 value, 16-bit position in
// the block), padded to the part's longest row so that no lane branches.  The copy engine keeps kBjStages chunks
// ahead of the sweep, so a level costs only shared-memory latencies; a row's
// packed data is read one and two parts ahead, which leaves the gather of y,
// the multiply-add chain and one barrier between two levels.  W warps sweep: one,
// without any block barrier, where levels hold up to 32 rows on average or where
// whole chunks would be half empty; the other warps only load and store the block's
// vector.
// 64^3, 112 blocks, both factors (272 levels): 41 us, where one launch a factor
// reading it from L2 level by level took 453 us.  What is left is the sweep's own
// chain, 0.15 us a level.  (A row's groups are not unrolled where one warp sweeps: 41
// against 45 us; several warps: 222 against 211 us at 16 blocks.)
// The in-place vector y holds the right-hand side, then L^-1 in, then the
// result; the terms and roundings of a row are k_trsv_bj's.
// ---------------------------------------------------------------------------
constexpr int kBjChunk = 16384, kBjStages = 4, kBjThreads = 256, kBjMaxWarps = 8;
constexpr int kBjPadLimit = 4;  // most words packed for every word the factors need
constexpr int32_t kIluSmemRows = 48 * 1024;  // longest block: fp16 vector of 96 KB, 16-bit positions

// Where one warp sweeps, chunks hold what is used of them, and a stage the largest
// of them, so that many small blocks cost neither memory nor bandwidth (64^3, 32,768
// blocks of 8 rows: 1.2 GB and 88.0 ms a solve with whole chunks, 174 MB and 20.1 ms).
// Several warps sweep blocks of many whole chunks; copies of a constant size are 5
// to 7% faster there (16 blocks at 64^3: 211 us an application, 222 with sizes read
// from memory).
struct BjStream {
  const unsigned char *chunks = nullptr;  // one warp: chunk c from chunk_at[c] * 16 bytes on; several: from c * kBjChunk on
  const int32_t *chunk_at = nullptr;      // (chunks + 1)
  const int32_t *blk_chunk = nullptr;     // per block: first chunk (nblocks + 1); lower chunks, then upper ones
  const int32_t *blk_pos = nullptr;       // per block: first vector position (nblocks + 1)
  int32_t warps = 1;                      // sweeping warps
  int32_t max_rows = 0;
  int32_t slot = kBjChunk;                // bytes of a stage
  // kBjThreads, or as many as the longest block has rows (whole warps): the loops over a block's vector step by kBjThreads
  int32_t threads() const { return std::max(warps * 32, std::min(kBjThreads, (max_rows + 31) / 32 * 32)); }
  size_t smem() const { return y_bytes() + (size_t)kBjStages * (slot + sizeof(uint64_t)) + 16; }
  __host__ __device__ size_t y_bytes() const { return ((size_t)(max_rows + 1) * sizeof(__half) + 127) / 128 * 128; }
};

// Chunk: 4 words {parts, 0, 0, 0}; 2 words a part; 1 word a row; the entries,
// from a 16-byte boundary, in groups of 4 words, a part's first groups row by
// row, then its second ones ...: every row of a part has the part's groups.
//   part word 0: first row word (from the chunk) | rows << 16; word 1: first group (16-byte units) | groups << 16
//   row word: position | fp16 1/u_ii (1 in L) << 16
//   entry word: position | fp16 -value << 16; padding entries are -0 times the zero kept behind the block's vector
//   (which leaves every sum as it is, a negative zero too)
template <bool MULTI>
__global__ void __launch_bounds__(kBjThreads) k_bj_stream(BjStream T, const __half *__restrict__ in,
                                                          __half *__restrict__ out, const __half *__restrict__ ome,
                                                          int *err) {
  extern __shared__ __align__(128) unsigned char bj_smem[];
  __half *y = reinterpret_cast<__half *>(bj_smem);
  unsigned char *ring = bj_smem + T.y_bytes();
  uint64_t *bars = reinterpret_cast<uint64_t *>(ring + (size_t)kBjStages * (MULTI ? kBjChunk : T.slot));
  volatile int *gave_up = reinterpret_cast<volatile int *>(bars + kBjStages);
  const int b = blockIdx.x;
  const int c0 = T.blk_chunk[b], c1 = T.blk_chunk[b + 1];
  const int32_t p0 = T.blk_pos[b], len = T.blk_pos[b + 1] - p0;
  const int slot = MULTI ? kBjChunk : T.slot;
  auto fetch = [&](int c, int64_t at, int64_t to) {  // units at to `to`
    const int st = (c - c0) % kBjStages;
    const uint32_t bytes = MULTI ? kBjChunk : (uint32_t)(to - at) * 16;
    fence_proxy_async_smem();
    mbar_arrive_expect_tx(&bars[st], bytes);
    bulk_g2s(ring + (size_t)st * slot, T.chunks + (MULTI ? (size_t)c * kBjChunk : (size_t)at * 16), bytes, &bars[st]);
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < kBjStages; s++) mbar_init(&bars[s], 1);
    *gave_up = 0;
    fence_mbar_init();
    for (int c = c0; c < min(c1, c0 + kBjStages); c++) fetch(c, MULTI ? 0 : T.chunk_at[c], MULTI ? 0 : T.chunk_at[c + 1]);
  }
#pragma unroll 8
  for (int i = threadIdx.x; i < len; i += kBjThreads) y[i] = in[p0 + i];
  if (threadIdx.x == 0) y[len] = __ushort_as_half((unsigned short)0);  // what padding entries multiply
  __syncthreads();
  const int width = MULTI ? T.warps * 32 : 32;
  const int tid = threadIdx.x;
  if (tid < width) {
    auto sync = [&]() {
      if (MULTI) asm volatile("bar.sync 1, %0;" ::"r"(width) : "memory");
      else __syncwarp();
    };
    int c = c0;
    for (; c < c1; c++) {
      const int st = (c - c0) % kBjStages;
      const bool ok = mbar_wait_bounded(&bars[st], (uint32_t)(((c - c0) / kBjStages) & 1));
      if (!ok) *gave_up = 1;
      sync();
      if (*gave_up) break;
      const uint32_t *ch = reinterpret_cast<const uint32_t *>(ring + (size_t)st * slot);
      const int np = ch[0];
      int32_t n0 = 0, n1 = 0;
      if (!MULTI && tid == 0 && c + kBjStages < c1) {
        n0 = T.chunk_at[c + kBjStages];
        n1 = T.chunk_at[c + kBjStages + 1];
      }
      const uint2 *parts = reinterpret_cast<const uint2 *>(ch + 4);
      const uint4 *ent = reinterpret_cast<const uint4 *>(ch);
      auto half_of = [&](uint32_t bits) { return __ushort_as_half((unsigned short)bits); };
      // row l of part d: m its word, e its first group; stored where live
      auto row = [&](const uint2 d, int l, uint32_t m, uint4 e, bool live) {
        const int nr = d.x >> 16, ng = d.y >> 16;
        float t = __half2float(y[m & 0xffffu]);
#pragma unroll(MULTI ? 4 : 1)
        for (int g = 0; g < ng; g++) {
          const uint32_t w[4] = {e.x, e.y, e.z, e.w};
          __half v[4];
#pragma unroll
          for (int u = 0; u < 4; u++) v[u] = y[w[u] & 0xffffu];
          if (g + 1 < ng) e = ent[(d.y & 0xffffu) + (g + 1) * nr + l];
#pragma unroll
          for (int u = 0; u < 4; u++) t = fma_vx<float>(half_of(w[u] >> 16), v[u], t);
        }
        if (live) y[m & 0xffffu] = __float2half_rn(t * __half2float(half_of(m >> 16)));
      };
      // part words are read two parts ahead, this thread's row word and first
      // group one (threads past a part's rows repeat its last row, unstored; a part
      // without entries starts at 0, and the chunk is long enough for the read)
      auto lane_row = [&](const uint2 d) { return min(tid, (int)(d.x >> 16) - 1); };
      uint2 d0 = parts[0], d1 = parts[min(1, np - 1)];
      int l0 = lane_row(d0);
      uint32_t m0 = ch[(d0.x & 0xffffu) + l0];
      uint4 e0 = ent[(d0.y & 0xffffu) + l0];
      for (int q = 0; q < np; q++) {
        const uint2 d2 = parts[min(q + 2, np - 1)];
        const int l1 = lane_row(d1);
        const uint32_t m1 = ch[(d1.x & 0xffffu) + l1];
        const uint4 e1 = ent[(d1.y & 0xffffu) + l1];
        const int nr = d0.x >> 16;
        row(d0, l0, m0, e0, tid < nr);
        for (int r = tid + width; r < nr; r += width)  // a part without entries has no groups to read
          row(d0, r, ch[(d0.x & 0xffffu) + r], ent[(d0.y & 0xffffu) + (d0.y >> 16 ? r : 0)], true);
        sync();
        d0 = d1;
        d1 = d2;
        l0 = l1;
        m0 = m1;
        e0 = e1;
      }
      // every thread is past its reads of this stage: refill it
      if (tid == 0 && c + kBjStages < c1) fetch(c + kBjStages, n0, n1);
    }
    if (c < c1 && tid == 0) {
      atomicCAS(err, 0, (int)DEV_TIMEOUT_TRSV);
      // let the copies in flight land before the block's shared memory goes (bounded)
      for (int k = c; k < min(c1, c + kBjStages); k++)
        mbar_wait_bounded(&bars[(k - c0) % kBjStages], (uint32_t)(((k - c0) / kBjStages) & 1));
    }
  }
  __syncthreads();
  // the reference solves, then scales: hout *= ome[0] (work/src/f3r.cpp:216, 229)
  const float om = ome ? __half2float(*ome) : 1.0f;
  for (int i = threadIdx.x; i < len; i += kBjThreads)
    out[p0 + i] = ome ? __float2half_rn(__half2float(y[i]) * om) : y[i];
}

struct IluDevice {
  IluTri L, U;      // where the blocks cannot be streamed
  BjStream stream;  // max_rows > 0: the fused solve
  int32_t nblocks = 0;
  std::vector<void *> allocs;

  template <typename T> cudaError_t up(T **d, const std::vector<T> &h) {
    cudaError_t e = cudaMalloc((void **)d, sizeof(T) * std::max<size_t>(h.size(), 1));
    if (e != cudaSuccess) return e;
    allocs.push_back((void *)*d);
    return cudaMemcpy(*d, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice);
  }
  void release() {
    for (void *p : allocs) cudaFree(p);
    allocs.clear();
  }

  // levels of one triangular factor inside each block-Jacobi block
  static void levels(const HostCSR &M, bool upper, const std::vector<int32_t> &bptr, std::vector<int32_t> &order,
                     std::vector<int32_t> &lvl_off, std::vector<int32_t> &blk_lvl, int32_t &maxlev) {
    const int32_t n = M.n, nb = (int32_t)bptr.size() - 1;
    std::vector<int32_t> lev(n, 0);
    order.clear();
    lvl_off.assign(1, 0);
    blk_lvl.assign(1, 0);
    maxlev = 0;
    for (int32_t b = 0; b < nb; b++) {
      int32_t nl = 0;
      if (!upper) {
        for (int32_t i = bptr[b]; i < bptr[b + 1]; i++) {
          int32_t lv = 0;
          for (int32_t j = M.rptr[i]; j < M.rptr[i + 1]; j++)
            if (M.idx[j] < i) lv = std::max(lv, lev[M.idx[j]] + 1);
          lev[i] = lv;
          nl = std::max(nl, lv + 1);
        }
      } else {
        for (int32_t i = bptr[b + 1] - 1; i >= bptr[b]; i--) {
          int32_t lv = 0;
          for (int32_t j = M.rptr[i]; j < M.rptr[i + 1]; j++)
            if (M.idx[j] > i) lv = std::max(lv, lev[M.idx[j]] + 1);
          lev[i] = lv;
          nl = std::max(nl, lv + 1);
        }
      }
      // bucket the block's rows by level
      std::vector<int32_t> cnt(nl + 1, 0);
      for (int32_t i = bptr[b]; i < bptr[b + 1]; i++) cnt[lev[i] + 1]++;
      for (int32_t l = 0; l < nl; l++) cnt[l + 1] += cnt[l];
      const size_t base = order.size();
      order.resize(base + (bptr[b + 1] - bptr[b]));
      std::vector<int32_t> fill(cnt.begin(), cnt.end() - 1);
      for (int32_t i = bptr[b]; i < bptr[b + 1]; i++) order[base + fill[lev[i]]++] = i;
      for (int32_t l = 0; l < nl; l++) lvl_off.push_back((int32_t)(base + cnt[l + 1]));
      blk_lvl.push_back(blk_lvl.back() + nl);
      maxlev = std::max(maxlev, nl);
    }
  }

  // a factor in the order the kernels visit it: rows by block and level, a
  // row's off-diagonal entries in processing order (increasing columns for L,
  // decreasing for U)
  struct TriHost {
    std::vector<int32_t> order, lvl_off, blk_lvl, idx;
    std::vector<int4> meta;
    std::vector<double> val, dinv;
  };
  static void visit_order(TriHost &t, const HostCSR &M, bool upper, const std::vector<int32_t> &bptr,
                          const std::vector<int32_t> &pos) {
    int32_t nlevels = 0;
    levels(M, upper, bptr, t.order, t.lvl_off, t.blk_lvl, nlevels);
    const size_t nq = t.order.size();
    t.meta.resize(nq);
    t.val.reserve(M.val.size());
    t.idx.reserve(M.idx.size());
    if (upper) t.dinv.resize(nq);
    for (size_t q = 0; q < nq; q++) {
      const int32_t i = t.order[q], r0 = M.rptr[i], r1 = M.rptr[i + 1];
      t.meta[q].x = pos[i];
      t.meta[q].y = (int32_t)t.idx.size();
      if (!upper) {
        for (int32_t j = r0; j < r1 - 1; j++) {  // last entry is the unit diagonal
          t.val.push_back(M.val[j]);
          t.idx.push_back(pos[M.idx[j]]);
        }
      } else {
        for (int32_t j = r1 - 1; j > r0; j--) {  // first entry is the diagonal
          t.val.push_back(M.val[j]);
          t.idx.push_back(pos[M.idx[j]]);
        }
        t.dinv[q] = 1.0 / M.val[r0];
      }
      t.meta[q].z = (int32_t)t.idx.size();
      t.meta[q].w = 0;
    }
  }

  Status upload_tri(IluTri &T, const TriHost &h, bool upper) {
    if (up(&T.meta, h.meta) != cudaSuccess || up(&T.idx, h.idx) != cudaSuccess ||
        up(&T.lvl_off, h.lvl_off) != cudaSuccess || up(&T.blk_lvl, h.blk_lvl) != cudaSuccess)
      return fail(F3R_ERROR_CUDA, "ILU upload failed");
    // fp16 values rounded once from fp64 (the reference casts CSR<double> to CSR<__half>, csr.hpp:23-25)
    F3R_TRY(to_half(&T.val, h.val));
    if (upper) F3R_TRY(to_half(&T.dinv, h.dinv));
    return F3R_SUCCESS;
  }

  Status to_half(__half **d, const std::vector<double> &v);
  // v rounded to fp16 as the device rounds it
  Status half_bits(std::vector<uint16_t> &h, const std::vector<double> &v) {
    __half *d = nullptr;
    F3R_TRY(to_half(&d, v));
    h.resize(v.size());
    const cudaError_t e = v.empty() ? cudaSuccess : cudaMemcpy(h.data(), d, v.size() * 2, cudaMemcpyDeviceToHost);
    cudaFree(d);
    allocs.pop_back();
    return e == cudaSuccess ? F3R_SUCCESS : fail(F3R_ERROR_CUDA, "ILU values");
  }

  // Appends one factor of block b (len rows from position p0) to the block's
  // chunks (see k_bj_stream), and where each starts to start.  false when a row does not fit a chunk.
  static bool pack_block(std::vector<uint32_t> &out, std::vector<size_t> &start, const TriHost &t, const std::vector<uint16_t> &val,
                         const std::vector<uint16_t> &dinv, bool upper, int32_t b, int32_t p0, int32_t len) {
    constexpr int kWords = kBjChunk / 4;
    auto up4 = [](int x) { return (x + 3) & ~3; };
    struct Part {
      std::vector<int32_t> rows;
      int groups = 0;
    };
    std::vector<Part> parts;
    auto groups_of = [&](int32_t q) { return (t.meta[q].z - t.meta[q].y + 3) / 4; };
    int nrows = 0, closed = 0;  // rows of the chunk; entry words of its complete parts
    auto fits = [&](int np, int nr, int entries) { return 4 + 2 * np + up4(nr + (2 * np & 2)) + 4 + entries <= kWords; };
    auto flush = [&]() {
      if (parts.empty()) return;
      const size_t base = out.size();
      const int np = (int)parts.size();
      int rw = 4 + 2 * np, at = up4(rw + nrows), end = at;
      for (const Part &pt : parts) end += 4 * pt.groups * (int)pt.rows.size();
      for (const Part &pt : parts)  // the kernel reads a group ahead for every swept row of a part, also where it has none
        if (pt.groups == 0) end = std::max(end, 4 * std::min((int)pt.rows.size(), kBjMaxWarps * 32));
      start.push_back(base);
      out.resize(base + end, 0u);
      uint32_t *c = out.data() + base;
      c[0] = (uint32_t)np;
      for (int q = 0; q < np; q++) {
        const Part &pt = parts[q];
        const int nr = (int)pt.rows.size();
        c[4 + 2 * q] = (uint32_t)rw | ((uint32_t)nr << 16);
        c[4 + 2 * q + 1] = (pt.groups ? (uint32_t)(at / 4) : 0u) | ((uint32_t)pt.groups << 16);
        for (int r = 0; r < nr; r++) {
          const int4 m = t.meta[pt.rows[r]];
          c[rw + r] = (uint32_t)(m.x - p0) | ((upper ? (uint32_t)dinv[pt.rows[r]] : 0x3C00u) << 16);
          for (int k = 0; k < 4 * pt.groups; k++) {
            const int32_t j = m.y + k;
            c[at + ((k / 4) * nr + r) * 4 + k % 4] =
                j < m.z ? (uint32_t)(t.idx[j] - p0) | ((uint32_t)(val[j] ^ 0x8000u) << 16) : (uint32_t)len | 0x80000000u;
          }
        }
        rw += nr;
        at += 4 * nr * pt.groups;
      }
      parts.clear();
      nrows = 0;
      closed = 0;
    };
    for (int32_t l = t.blk_lvl[b]; l < t.blk_lvl[b + 1]; l++) {
      bool open = false;  // this level's part in the chunk
      for (int32_t q = t.lvl_off[l]; q < t.lvl_off[l + 1]; q++) {
        const int g = groups_of(q);
        if (!fits(1, 1, 4 * g)) return false;
        if (open) {
          Part &pt = parts.back();
          const int ng = std::max(pt.groups, g);
          if (!fits((int)parts.size(), nrows + 1, closed + 4 * ng * ((int)pt.rows.size() + 1))) {
            flush();
            open = false;
          }
        } else if (!fits((int)parts.size() + 1, nrows + 1, closed + 4 * g)) {
          flush();
        }
        if (!open) {
          parts.emplace_back();
          open = true;
        }
        parts.back().rows.push_back(q);
        parts.back().groups = std::max(parts.back().groups, g);
        nrows++;
      }
      if (open) closed += 4 * parts.back().groups * (int)parts.back().rows.size();
    }
    flush();
    return true;
  }

  // the chunks of all blocks; stream.max_rows stays 0 where the blocks do not
  // occupy contiguous positions, a block or row is too large, or padding the parts
  // to their longest rows takes too much (kBjPadLimit)
  Status build_stream(const TriHost &l, const TriHost &u, const std::vector<int32_t> &bptr,
                      const std::vector<int32_t> &pos) {
    const int32_t nb = (int32_t)bptr.size() - 1;
    std::vector<int32_t> bpos(nb + 1, 0), first(nb + 1, 0);
    int32_t maxlen = 0;
    for (int32_t b = 0; b < nb; b++) {
      bpos[b] = bptr[b];
      maxlen = std::max(maxlen, bptr[b + 1] - bptr[b]);
      for (int32_t i = bptr[b]; i < bptr[b + 1]; i++)
        if (pos[i] != i) return F3R_SUCCESS;
    }
    bpos[nb] = bptr[nb];
    if (maxlen > kIluSmemRows) return F3R_SUCCESS;
    std::vector<uint16_t> lv, uv, ud;
    F3R_TRY(half_bits(lv, l.val));
    F3R_TRY(half_bits(uv, u.val));
    F3R_TRY(half_bits(ud, u.dinv));
    // words the rows' parts need without padding, chunk headers included
    const int64_t need = (int64_t)l.val.size() + (int64_t)u.val.size() + 6 * (int64_t)pos.size() + 16 * (int64_t)nb;
    std::vector<std::vector<uint32_t>> packed(nb);
    std::vector<std::vector<size_t>> starts(nb);
    int bad = 0;
    int64_t words = 0;
#pragma omp parallel for schedule(dynamic, 16) reduction(+ : bad, words)
    for (int32_t b = 0; b < nb; b++) {
      if (words > kBjPadLimit * need ||
          !pack_block(packed[b], starts[b], l, lv, ud, false, b, bpos[b], bpos[b + 1] - bpos[b]) ||
          !pack_block(packed[b], starts[b], u, uv, ud, true, b, bpos[b], bpos[b + 1] - bpos[b]))
        bad++;
      words += (int64_t)packed[b].size();
    }
    if (bad || words > kBjPadLimit * need || words > (int64_t)INT32_MAX * 4) return F3R_SUCCESS;
    // warps by the mean rows of a level; one warp needs no block barrier
    const int64_t lev = (int64_t)l.lvl_off.size() + (int64_t)u.lvl_off.size() - 2;
    const int64_t avg = lev > 0 ? 2 * (int64_t)l.order.size() / lev : 0;
    size_t nchunks = 0;
    for (const auto &st : starts) nchunks += st.size();
    const bool whole = avg > 32 && (int64_t)nchunks * (kBjChunk / 4) <= 2 * words;
    std::vector<uint32_t> all;
    all.reserve(whole ? nchunks * (kBjChunk / 4) : (size_t)words);
    std::vector<int32_t> at(1, 0);  // in 16-byte units
    int32_t slot = 16;
    for (int32_t b = 0; b < nb; b++) {
      for (size_t c = 0; c < starts[b].size(); c++) {
        const size_t c0 = starts[b][c], c1 = c + 1 < starts[b].size() ? starts[b][c + 1] : packed[b].size();
        slot = std::max(slot, (int32_t)(c1 - c0) * 4);
        all.insert(all.end(), packed[b].begin() + c0, packed[b].begin() + c1);
        if (whole) all.resize((size_t)(first[b] + c + 1) * (kBjChunk / 4), 0u);
        at.push_back((int32_t)(all.size() / 4));
      }
      first[b + 1] = first[b] + (int32_t)starts[b].size();
      std::vector<uint32_t>().swap(packed[b]);
    }
    uint32_t *d = nullptr;
    int32_t *fd = nullptr, *pd = nullptr, *ad = nullptr;
    if (up(&d, all) != cudaSuccess || up(&fd, first) != cudaSuccess || up(&pd, bpos) != cudaSuccess ||
        up(&ad, at) != cudaSuccess)
      return fail(F3R_ERROR_OUT_OF_MEMORY, "ILU upload failed");
    stream.chunks = reinterpret_cast<const unsigned char *>(d);
    stream.chunk_at = ad;
    stream.slot = whole ? kBjChunk : slot;
    stream.warps = whole ? (int32_t)std::min<int64_t>(kBjMaxWarps, (avg + 31) / 32) : 1;
    stream.blk_chunk = fd;
    stream.blk_pos = pd;
    stream.max_rows = std::max(maxlen, 1);
    return F3R_SUCCESS;
  }

  Status build(cudaStream_t, const HostCSR &Lh, const HostCSR &Uh, const std::vector<int32_t> &perm, bool permuted,
               const std::vector<int32_t> &bptr) {
    const int32_t n = Lh.n;
    std::vector<int32_t> pos(n);
    for (int32_t i = 0; i < n; i++) pos[i] = i;
    if (permuted)
      for (int32_t s = 0; s < n; s++) pos[perm[s]] = s;
    nblocks = (int32_t)bptr.size() - 1;
    TriHost l, u;
    visit_order(l, Lh, false, bptr, pos);
    visit_order(u, Uh, true, bptr, pos);
    F3R_TRY(build_stream(l, u, bptr, pos));
    if (stream.max_rows > 0) {
      // the attribute is the kernel's, shared by every solver: always the cap
      BjStream cap;
      cap.max_rows = kIluSmemRows;
      if (cudaFuncSetAttribute(k_bj_stream<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap.smem()) !=
              cudaSuccess ||
          cudaFuncSetAttribute(k_bj_stream<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap.smem()) !=
              cudaSuccess)
        return fail(F3R_ERROR_CUDA, "ILU shared-memory attribute");
      return F3R_SUCCESS;
    }
    F3R_TRY(upload_tri(L, l, false));
    return upload_tri(U, u, true);
  }

  int launches() const { return stream.max_rows > 0 ? 1 : 2; }  // kernels of one apply

  // out = U^-1 L^-1 x (tmp: scratch); ome (nullable) scales the result
  Status apply(cudaStream_t st, const __half *x, __half *tmp, __half *out, const __half *ome, int *err) const {
    if (nblocks == 0) return F3R_SUCCESS;
    if (stream.max_rows > 0) {
      const int threads = stream.threads();
      if (stream.warps > 1) k_bj_stream<true><<<nblocks, threads, stream.smem(), st>>>(stream, x, out, ome, err);
      else k_bj_stream<false><<<nblocks, threads, stream.smem(), st>>>(stream, x, out, ome, err);
    } else {
      k_trsv_bj<false><<<nblocks, 256, 0, st>>>(L, x, tmp, nullptr);
      k_trsv_bj<true><<<nblocks, 256, 0, st>>>(U, tmp, out, ome);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(F3R_ERROR_CUDA, std::string("ILU trsv launch: ") + cudaGetErrorString(e));
    return F3R_SUCCESS;
  }
};

// ---------------------------------------------------------------------------
// Global ILU(0), level-scheduled over the whole GPU (F3R_PRECOND_ILU0_LEVEL).
//
// One factor of the global (single-block) ILU(0) is solved by one kernel
// without grid barriers.  The rows are listed level by level, every level
// padded with -1 to whole 32-row chunks, so the 32 rows of a chunk never read
// each other.  Warps take chunks in list order from an atomic counter; a row
// waits until each row it reads carries this launch's generation in its flag
// (acquire load), then computes exactly as k_trsv_bj does (same order of
// terms, same roundings) and publishes value then flag (release store).  A
// warp waits only on chunks taken before its own by running warps, and the
// lowest unfinished chunk never waits, so the solve always completes.  Every
// wait is bounded (kWaitLimitNs); the first timeout sets the device error
// word, which ends every other wait of the launch at once.  The last block to
// finish resets the counter and advances the generation, so back-to-back
// launches (and graph replays) need no host work.
struct IluLevelTri {
  // rows level by level, padded to 32-row chunks, in the order warps take them
  int4 *meta = nullptr;     // per slot: vector position (-1: padding), first and end entry
  __half *val = nullptr;    // entries in processing order (diagonal excluded)
  int32_t *idx = nullptr;   // their columns, mapped to vector positions
  __half *dinv = nullptr;   // upper only: per slot
  int32_t nchunks = 0;
  int32_t nlevels = 0;
  int32_t *flag = nullptr;                  // per vector position: generation of its last write
  unsigned int *state = nullptr;            // chunk counter, finished-block ticket, generation
};

__device__ __forceinline__ unsigned int ld_relaxed_u32(const int32_t *p) {
  unsigned int v;
  asm volatile("ld.relaxed.gpu.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_u32(int32_t *p, unsigned int v) {
  asm volatile("st.release.gpu.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

constexpr int kLevelBatch = 16;  // dependencies polled, then read, together

// Waits until flag[q[u]] == gen for every u < cnt (relaxed polls, then one
// fence orders the caller's later loads after them).  Bounded: after
// limit_ns of %globaltimer it records DEV_TIMEOUT_TRSV in *err and returns
// false; it also returns false at once when *err is already set (another
// wait of the launch gave up, or the solve broke down), so no wait outlives
// the first failure by more than one bound.
__device__ __forceinline__ bool wait_flags(const int32_t *flag, const int32_t (&q)[kLevelBatch], int cnt,
                                           unsigned int gen, int *err, unsigned long long limit_ns) {
  volatile int *verr = err;
  uint32_t waiting = (1u << cnt) - 1u;
  unsigned long long t0 = 0;
  int polls = 0;
  bool ok = true;
  while (true) {
#pragma unroll
    for (int u = 0; u < kLevelBatch; u++)
      if ((waiting >> u) & 1u)
        if (ld_relaxed_u32(flag + q[u]) == gen) waiting &= ~(1u << u);
    if (waiting == 0) break;
    if (*verr != 0) {
      ok = false;
      break;
    }
    if (polls++ == 0) t0 = global_ns();
    else if (global_ns() - t0 > limit_ns) {
      atomicCAS(err, 0, (int)DEV_TIMEOUT_TRSV);
      ok = false;
      break;
    }
    if (polls > 4) __nanosleep(32);
  }
  __threadfence();
  return ok;
}

template <bool UPPER>
__global__ void __launch_bounds__(256, 2) k_trsv_level(IluLevelTri T, const __half *__restrict__ in, __half *out,
                                                    int *err) {
  __shared__ unsigned int gen_s;
  if (threadIdx.x == 0) gen_s = *(volatile unsigned int *)&T.state[2] + 1u;
  __syncthreads();
  const unsigned int gen = gen_s;
  const int lane = threadIdx.x & 31;
  bool abort = false;
  while (true) {
    unsigned int c = 0;
    if (lane == 0) c = atomicAdd(&T.state[0], 1u);
    c = __shfl_sync(0xffffffffu, c, 0);
    if (c >= (unsigned int)T.nchunks) break;
    const size_t slot = (size_t)c * 32 + lane;
    const int4 m = T.meta[slot];
    if (m.x >= 0) {
      const int32_t p = m.x;
      float t = __half2float(in[p]);
      // the entries in processing order: lower by increasing, upper by decreasing column
      const int32_t b = m.y, ndep = m.z - m.y;
      for (int32_t base = 0; base < ndep; base += kLevelBatch) {
        const int cnt = min(kLevelBatch, ndep - base);
        int32_t q[kLevelBatch];
        float lv[kLevelBatch];
#pragma unroll
        for (int u = 0; u < kLevelBatch; u++)
          if (u < cnt) {
            const int32_t j = b + base + u;
            q[u] = T.idx[j];
            lv[u] = __half2float(T.val[j]);
          }
        // every flag of the batch polled at once; one fence orders the value loads after them
        if (!abort) abort = !wait_flags(T.flag, q, cnt, gen, err, kWaitLimitNs);
        float y[kLevelBatch];
#pragma unroll
        for (int u = 0; u < kLevelBatch; u++)
          if (u < cnt) y[u] = __half2float(__ldcg(out + q[u]));
#pragma unroll
        for (int u = 0; u < kLevelBatch; u++)
          if (u < cnt) t = __fmaf_rn(-lv[u], y[u], t);
      }
      const __half h = UPPER ? __float2half_rn(t * __half2float(T.dinv[slot])) : __float2half_rn(t);
      out[p] = h;
      __threadfence();
      st_release_u32(T.flag + p, gen);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned int tk = atomicAdd(&T.state[1], 1u);
    if (tk == gridDim.x - 1) {
      T.state[0] = 0;
      T.state[1] = 0;
      __threadfence();
      atomicAdd(&T.state[2], 1u);
    }
  }
}

struct IluLevel {
  IluLevelTri L, U;
  int grid = 0, scale_grid = 1;
  int64_t n = 0;
  std::vector<void *> allocs;

  template <typename T> cudaError_t up(T **d, const std::vector<T> &h) {
    cudaError_t e = cudaMalloc((void **)d, sizeof(T) * std::max<size_t>(h.size(), 1));
    if (e != cudaSuccess) return e;
    allocs.push_back((void *)*d);
    return cudaMemcpy(*d, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice);
  }
  void release() {
    for (void *p : allocs) cudaFree(p);
    allocs.clear();
  }

  Status build_tri(IluLevelTri &T, const HostCSR &M, bool upper, const std::vector<int32_t> &pos) {
    const int32_t n = M.n;
    std::vector<int32_t> order, lvl_off, blk_lvl;
    int32_t nl = 0;
    IluDevice::levels(M, upper, std::vector<int32_t>{0, n}, order, lvl_off, blk_lvl, nl);
    std::vector<int32_t> padded;
    padded.reserve(order.size() + (size_t)nl * 32);
    for (int32_t l = 0; l + 1 < (int32_t)lvl_off.size(); l++) {
      for (int32_t q = lvl_off[l]; q < lvl_off[l + 1]; q++) padded.push_back(order[q]);
      while (padded.size() % 32) padded.push_back(-1);
    }
    T.nchunks = (int32_t)(padded.size() / 32);
    T.nlevels = nl;
    // the factor in slot order; fp16 values rounded once from fp64
    std::vector<int4> meta(padded.size());
    std::vector<double> v, dinv(upper ? padded.size() : 0, 1.0);
    std::vector<int32_t> idx;
    v.reserve(M.val.size());
    idx.reserve(M.idx.size());
    for (size_t q = 0; q < padded.size(); q++) {
      const int32_t i = padded[q];
      meta[q] = make_int4(-1, 0, 0, 0);
      if (i < 0) continue;
      const int32_t r0 = M.rptr[i], r1 = M.rptr[i + 1];
      meta[q].x = pos[i];
      meta[q].y = (int32_t)idx.size();
      if (!upper) {
        for (int32_t j = r0; j < r1 - 1; j++) {  // last entry is the unit diagonal
          v.push_back(M.val[j]);
          idx.push_back(pos[M.idx[j]]);
        }
      } else {
        for (int32_t j = r1 - 1; j > r0; j--) {  // first entry is the diagonal
          v.push_back(M.val[j]);
          idx.push_back(pos[M.idx[j]]);
        }
        dinv[q] = 1.0 / M.val[r0];
      }
      meta[q].z = (int32_t)idx.size();
    }
    const std::vector<int32_t> zeros(std::max(n, 1), 0);
    const std::vector<unsigned int> st(3, 0u);
    if (up(&T.meta, meta) != cudaSuccess || up(&T.idx, idx) != cudaSuccess || up(&T.flag, zeros) != cudaSuccess ||
        up(&T.state, st) != cudaSuccess)
      return fail(F3R_ERROR_CUDA, "ILU upload failed");
    F3R_TRY(half_copy(&T.val, v));
    if (upper) F3R_TRY(half_copy(&T.dinv, dinv));
    return F3R_SUCCESS;
  }

  Status half_copy(__half **d, const std::vector<double> &v);

  Status build(int sm_count, const HostCSR &Lh, const HostCSR &Uh, const std::vector<int32_t> &perm, bool permuted) {
    const int32_t n = Lh.n;
    this->n = n;
    scale_grid = (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, (int64_t)sm_count * 8));
    std::vector<int32_t> pos(n);
    for (int32_t i = 0; i < n; i++) pos[i] = i;
    if (permuted)
      for (int32_t s = 0; s < n; s++) pos[perm[s]] = s;
    F3R_TRY(build_tri(L, Lh, false, pos));
    F3R_TRY(build_tri(U, Uh, true, pos));
    // warps for about four levels' chunks at a time: the frontier has work for
    // them, and few enough are left spinning ahead of it
    const int64_t chunks = std::max(L.nchunks, U.nchunks), levels = std::max(1, std::max(L.nlevels, U.nlevels));
    const int64_t warps = 4 * ((chunks + levels - 1) / levels);
    grid = (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)sm_count * 2, (warps + 7) / 8));
    return F3R_SUCCESS;
  }

  // out = U^-1 L^-1 x (tmp holds L^-1 x); ome (nullable) scales the result
  Status apply(cudaStream_t st, const __half *x, __half *tmp, __half *out, const __half *ome, int *err) const {
    k_trsv_level<false><<<grid, 256, 0, st>>>(L, x, tmp, err);
    k_trsv_level<true><<<grid, 256, 0, st>>>(U, tmp, out, err);
    // then the scaling, as the reference: hout *= ome[0] (work/src/f3r.cpp:216, 229)
    if (ome) k_half_scale<<<scale_grid, 256, 0, st>>>(out, ome, n);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(F3R_ERROR_CUDA, std::string("ILU trsv launch: ") + cudaGetErrorString(e));
    return F3R_SUCCESS;
  }
};

// The level solve's flag wait on one flag (f3r_context_wait_probe): the
// flag holds gen when set, 0 otherwise.
__global__ void k_wait_probe(const int32_t *flag, unsigned int gen, int *err, unsigned long long limit_ns) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  int32_t q[kLevelBatch] = {0};
  wait_flags(flag, q, 1, gen, err, limit_ns);
}

}  // namespace f3r
