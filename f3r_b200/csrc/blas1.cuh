// blas1.cuh -- the Gram-Schmidt kernels of the single-column fp32 levels: the
// dot products of w with up to 8 basis vectors, and the update, norm and Givens
// step.
//
// They form exactly the sums of k_dotsK (blockdots.cuh) and k_cgs_updateK (block.cuh,
// the K-column kernels whose columns must equal single solves): a logical grid
// of up to 8 blocks of 256 threads an SM, each thread the 16-byte quads tid,
// tid + stride, ... in order; warp butterflies; the 8 warps of a block in order;
// then the blocks by thread t = t, t + 256, ..., butterfly, warps.  What differs
// is who computes them: a block here works L = 2 logical blocks where there are
// more than half a wave of them, with 64 registers a thread instead of 32 and
// nothing spilled, twice the loads in flight a thread, all values of a warp
// reduced at once, and the small arrays of the Givens step read ahead by the
// whole block.  Two more things save bytes and time:
//  * a basis vector is not normalised in place: its factor 1/h (VecScale) is
//    multiplied in by whoever reads it, the rounding the stored vector had;
//  * up to 8 dots take one pass over w (two of 4 before).
// In the solves, us a call (before -> here; hot, so partly from L2):
//   dots, nv <= 4    16^3 3.9 -> 3.2   95x83x71 6.5 -> 4.5    192^3 27.0 -> 18.9 (99 MB: 5.2 TB/s)
//   dots, nv 5..8    16^3 5.6 -> 4.1   95x83x71 9.5 -> 6.0    192^3 54.5 -> 45.1
//   update, nv <= 4  16^3 5.2 -> 4.6   95x83x71 7.1 -> 6.0    192^3 24.9 -> 19.8 (127 MB: 6.4 TB/s)
//   R's entry (one write of w fewer)                          192^3 11.1 -> 9.2
//   x = Z y, fp16 Z  16^3 2.1 -> 1.9   95x83x71 3.7 -> 3.0    192^3 17.2 -> 13.0
// On small systems what is left is launch, two trips to L2 and the serial
// Givens step; on large ones the bytes.
#pragma once

#include "block.cuh"

namespace f3r {

constexpr int kMaxDots1 = 8;

// the vectors and their pending factors (null: none)
struct Basis8 {
  const float *p[kMaxDots1];
  const float *s[kMaxDots1];
};

// The butterfly sums (offsets 16, 8, 4, 2, 1) of M values of every lane at once,
// M a power of two up to 8: each of the first steps halves the values a lane
// carries.  Lane l ends with value index_of(l); every sum is the same tree of
// additions as warp_sum's.
template <int M> struct WarpSums {
  static constexpr int LOG = M == 1 ? 0 : M == 2 ? 1 : M == 4 ? 2 : 3;
  static __device__ __forceinline__ float run(float (&v)[M]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 0; d < LOG; d++) {
      const int o = 16 >> d, half = M >> (d + 1);
      const bool up = lane & o;
#pragma unroll
      for (int i = 0; i < half; i++) {
        const float send = up ? v[i] : v[i + half];
        const float keep = up ? v[i + half] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
    float t = v[0];
#pragma unroll
    for (int o = 16 >> LOG; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
  }
  static __device__ __forceinline__ int index_of(int lane) { return lane >> (5 - LOG); }
  // the lanes that write: one a value
  static __device__ __forceinline__ bool writes(int lane) { return (lane & ((32 >> LOG) - 1)) == 0; }
};

// thread 0's acquire-release increment between two block barriers: true in the
// last block, which then sees every block's partial sums
__device__ __forceinline__ bool last_block1(unsigned int *ticket) {
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned int t;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(t) : "l"(ticket) : "memory");
    last = t == gridDim.x - 1;
  }
  __syncthreads();
  return last;
}

// sums of the logical blocks' partials for M values (of ntot from q0 on): value
// q0 + i on thread i
template <int M>
__device__ __forceinline__ float final_sums1(const float *part, int lgrid, int q0, int nq, int ntot, float (&sw)[8][M]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int B = 5;  // all of a thread's blocks at 8 an SM
  float s[M];
#pragma unroll
  for (int i = 0; i < M; i++) s[i] = 0.0f;
  for (int b0 = threadIdx.x; b0 < lgrid; b0 += B * 256) {
    float v[B][M];
#pragma unroll
    for (int u = 0; u < B; u++)
#pragma unroll
      for (int i = 0; i < M; i++)
        if (b0 + u * 256 < lgrid && i < nq) v[u][i] = __ldcg(part + (size_t)(b0 + u * 256) * ntot + q0 + i);
#pragma unroll
    for (int u = 0; u < B; u++)
#pragma unroll
      for (int i = 0; i < M; i++)
        if (b0 + u * 256 < lgrid && i < nq) s[i] += v[u][i];
  }
  const float t = WarpSums<M>::run(s);
  if (WarpSums<M>::writes(lane)) sw[warp][WarpSums<M>::index_of(lane)] = t;
  __syncthreads();
  float r = 0.0f;
  if ((int)threadIdx.x < nq)
#pragma unroll
    for (int w = 0; w < 8; w++) r += sw[w][threadIdx.x];
  __syncthreads();
  return r;
}

// H(j, k) = <w, V(k)>, k < nv <= NV, all with the unmodified w (gmres.hpp:112-114)
template <int NV, int L>
__global__ void __launch_bounds__(256, 4)
    k_dots1(const float *w, Basis8 V, int nv, int64_t n, int lgrid, GridRed gr, float *hcol) {
  stream_order();
  __shared__ float sred[8][L * NV];
  __shared__ float sw[8][4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float a[L][NV], sc[NV];
#pragma unroll
  for (int k = 0; k < NV; k++) {
    sc[k] = k < nv && V.s[k] ? *V.s[k] : 1.0f;
#pragma unroll
    for (int l = 0; l < L; l++) a[l][k] = 0.0f;
  }
  const int64_t stride = (int64_t)lgrid * 256, nq = n / 4, q0 = (int64_t)blockIdx.x * L * 256 + threadIdx.x;
  for (int64_t q = q0; q < nq; q += stride) {
    float wv[L][4];
#pragma unroll
    for (int l = 0; l < L; l++)
      if (l == 0 || (q + l * 256 < nq && blockIdx.x * L + l < lgrid)) {
        const float4 t = ld_stream(reinterpret_cast<const float4 *>(w) + q + l * 256);
        wv[l][0] = t.x; wv[l][1] = t.y; wv[l][2] = t.z; wv[l][3] = t.w;
      }
#pragma unroll
    for (int k0 = 0; k0 < NV; k0 += 4) {
      float4 v[4][L];
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (k0 + k < NV && k0 + k < nv) {
#pragma unroll
          for (int l = 0; l < L; l++)
            if (l == 0 || (q + l * 256 < nq && blockIdx.x * L + l < lgrid))
              v[k][l] = ld_stream(reinterpret_cast<const float4 *>(V.p[k0 + k]) + q + l * 256);
        }
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (k0 + k < NV && k0 + k < nv) {
          const float s = sc[k0 + k];
#pragma unroll
          for (int l = 0; l < L; l++)
            if (l == 0 || (q + l * 256 < nq && blockIdx.x * L + l < lgrid)) {
              float x = a[l][k0 + k];
              x = __fmaf_rn(wv[l][0], mul_rn(v[k][l].x, s), x);
              x = __fmaf_rn(wv[l][1], mul_rn(v[k][l].y, s), x);
              x = __fmaf_rn(wv[l][2], mul_rn(v[k][l].z, s), x);
              x = __fmaf_rn(wv[l][3], mul_rn(v[k][l].w, s), x);
              a[l][k0 + k] = x;
            }
        }
    }
  }
  if (q0 < n - nq * 4) {  // the last n % 4 elements: the first threads of logical block 0
    const int64_t i = nq * 4 + q0;
    const float wi = w[i];
#pragma unroll
    for (int k = 0; k < NV; k++)
      if (k < nv) a[0][k] = __fmaf_rn(wi, mul_rn(V.p[k][i], sc[k]), a[0][k]);
  }
#pragma unroll
  for (int l = 0; l < L; l++) {
    const float t = WarpSums<NV>::run(a[l]);
    if (WarpSums<NV>::writes(lane)) sred[warp][l * NV + WarpSums<NV>::index_of(lane)] = t;
  }
  __syncthreads();
  float *part = static_cast<float *>(gr.partials);
  if ((int)threadIdx.x < L * NV) {
    const int l = threadIdx.x / NV, k = threadIdx.x % NV, b = blockIdx.x * L + l;
    if (k < nv && b < lgrid) {
      float s = 0.0f;
#pragma unroll
      for (int q = 0; q < 8; q++) s += sred[q][threadIdx.x];
      part[(size_t)b * nv + k] = s;
    }
  }
  if (!last_block1(gr.ticket)) return;
#pragma unroll
  for (int k0 = 0; k0 < NV; k0 += 4)
    if (k0 < nv) {
      const int m = min(4, nv - k0);
      const float t = final_sums1<4>(part, lgrid, k0, m, nv, sw);
      if ((int)threadIdx.x < m) hcol[k0 + threadIdx.x] = t;
    }
  if (threadIdx.x == 0) *gr.ticket = 0;
}

// The level's small arrays of a Givens step, read ahead by the block (one
// thread reading them entry by entry made several trips to L2); m <= 8
struct Givens8 {
  static constexpr int LD = kMaxDots1 + 1;
  float H[kMaxDots1 * LD], cs[kMaxDots1], sn[kMaxDots1], e[LD], y[kMaxDots1];
  // column c's arrays by 64 threads t; sh[k * pitch]: the step's dots
  __device__ __forceinline__ void stage(const LevelK<float> &L, int c, int j, int compute_y, const float *sh, int pitch,
                                        int t) {
    if (t <= j) {
      H[j * LD + t] = sh[t * pitch];
      e[t] = L.e[c * L.vs + t];
      if (t < j) {
        cs[t] = L.cs[c * L.vs + t];
        sn[t] = L.sn[c * L.vs + t];
      }
    }
    if (compute_y && t < 64) {
      const int q = t / 8, i = t % 8;
      if (q < j && i <= q) H[q * LD + i] = L.H[c * L.hs + q * L.ldh + i];
    }
  }
  // one thread, after a barrier
  __device__ __forceinline__ void step(const LevelK<float> &L, int c, int j, int compute_y, int *err, float nrm2) {
    const GivensCtl<float> g{H, cs, sn, e, y, L.inv + c, nullptr, LD, j, compute_y, err};
    givens_step<float>(g, nrm2);
    float *Hc = L.H + c * L.hs + (int64_t)j * L.ldh;
    for (int i = 0; i <= j + 1; i++) Hc[i] = H[j * LD + i];
    L.cs[c * L.vs + j] = cs[j];
    L.sn[c * L.vs + j] = sn[j];
    L.e[c * L.vs + j] = e[j];
    L.e[c * L.vs + j + 1] = e[j + 1];
    if (compute_y)
      for (int i = 0; i <= j; i++) L.y[c * L.vs + i] = y[i];
  }
};

// w -= sum_k H(j, k) V(k) (MULMV order), ||w||^2 -> h_{j+1,j}, 1/h (L.inv), the
// Givens rotation and, on the level's last step, y (gmres.hpp:115-121); nv = j + 1 <= 8
template <int NV, int L>
__global__ void __launch_bounds__(256, 4)
    k_cgs1(float *w, Basis8 V, int nv, int64_t n, int lgrid, GridRed gr, LevelK<float> Lv, int j,
           int compute_y, int *err) {
  stream_order();
  __shared__ float sh[kMaxDots1], ssc[kMaxDots1];
  __shared__ float sred[8][L];
  __shared__ float sw[8][1];
  __shared__ Givens8 gs;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if ((int)threadIdx.x < nv) sh[threadIdx.x] = Lv.H[(int64_t)j * Lv.ldh + threadIdx.x];
#pragma unroll
  for (int k = 0; k < NV; k++)
    if (k < nv && (int)threadIdx.x == k) ssc[k] = V.s[k] ? *V.s[k] : 1.0f;
  const int64_t stride = (int64_t)lgrid * 256, nq = n / 4, q0 = (int64_t)blockIdx.x * L * 256 + threadIdx.x;
  float part[L];
#pragma unroll
  for (int l = 0; l < L; l++) part[l] = 0.0f;
  __syncthreads();
  for (int64_t q = q0; q < nq; q += stride) {
    float4 wv[L];
    float r[L][4];
    auto live = [&](int l) { return l == 0 || (q + l * 256 < nq && blockIdx.x * L + l < lgrid); };
#pragma unroll
    for (int l = 0; l < L; l++)
      if (live(l)) wv[l] = reinterpret_cast<const float4 *>(w)[q + l * 256];
#pragma unroll
    for (int k0 = 0; k0 < NV; k0 += 4) {
      float4 v[4][L];
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (k0 + k < nv) {
#pragma unroll
          for (int l = 0; l < L; l++)
            if (live(l)) v[k][l] = ld_stream(reinterpret_cast<const float4 *>(V.p[k0 + k]) + q + l * 256);
        }
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (k0 + k < nv) {
          const float h = sh[k0 + k], s = ssc[k0 + k];
#pragma unroll
          for (int l = 0; l < L; l++) {
            const float x[4] = {mul_rn(v[k][l].x, s), mul_rn(v[k][l].y, s), mul_rn(v[k][l].z, s), mul_rn(v[k][l].w, s)};
#pragma unroll
            for (int e = 0; e < 4; e++) r[l][e] = k0 + k == 0 ? mul_rn(x[e], h) : __fmaf_rn(x[e], h, r[l][e]);
          }
        }
    }
#pragma unroll
    for (int l = 0; l < L; l++)
      if (live(l)) {
        float x[4] = {sub_rn(wv[l].x, r[l][0]), sub_rn(wv[l].y, r[l][1]), sub_rn(wv[l].z, r[l][2]), sub_rn(wv[l].w, r[l][3])};
#pragma unroll
        for (int e = 0; e < 4; e++) part[l] = __fmaf_rn(x[e], x[e], part[l]);
        reinterpret_cast<float4 *>(w)[q + l * 256] = make_float4(x[0], x[1], x[2], x[3]);
      }
  }
  if (q0 < n - nq * 4) {
    const int64_t i = nq * 4 + q0;
    float r = mul_rn(mul_rn(V.p[0][i], ssc[0]), sh[0]);
#pragma unroll
    for (int k = 1; k < NV; k++)
      if (k < nv) r = __fmaf_rn(mul_rn(V.p[k][i], ssc[k]), sh[k], r);
    const float x = sub_rn(w[i], r);
    part[0] = __fmaf_rn(x, x, part[0]);
    w[i] = x;
  }
  const float t = WarpSums<L>::run(part);
  if (WarpSums<L>::writes(lane)) sred[warp][WarpSums<L>::index_of(lane)] = t;
  __syncthreads();
  float *parts = static_cast<float *>(gr.partials);
  if ((int)threadIdx.x < L && blockIdx.x * L + (int)threadIdx.x < lgrid) {
    float s = 0.0f;
#pragma unroll
    for (int q = 0; q < 8; q++) s += sred[q][threadIdx.x];
    parts[blockIdx.x * L + threadIdx.x] = s;
  }
  if (!last_block1(gr.ticket)) return;
  if (threadIdx.x < 64) gs.stage(Lv, 0, j, compute_y, sh, 1, threadIdx.x);
  const float nrm2 = final_sums1<1>(parts, lgrid, 0, 1, 1, sw);
  if (threadIdx.x == 0) {
    gs.step(Lv, 0, j, compute_y, err, nrm2);
    *gr.ticket = 0;
  }
}

// x = Z y of level 3 from its fp16 basis (gmres.hpp:127-128): 8 rows a thread,
// nz <= 8 columns, widened exactly, MULMV order
__global__ void __launch_bounds__(256) k_zy1(const __half *Z, int64_t ldz, const float *y, int nz, float *out,
                                             int64_t n) {
  stream_order();
  __shared__ float sy[kMaxDots1];
  if ((int)threadIdx.x < nz) sy[threadIdx.x] = y[threadIdx.x];
  __syncthreads();
  const int64_t q = (int64_t)blockIdx.x * 256 + threadIdx.x, i0 = q * 8;
  if (i0 + 8 <= n) {
    float r[8];
    for (int k0 = 0; k0 < nz; k0 += 4) {
      uint4 u[4];
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (k0 + k < nz) u[k] = ld_stream(reinterpret_cast<const uint4 *>(Z + (k0 + k) * ldz + i0));
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (k0 + k < nz) {
          const __half *z = reinterpret_cast<const __half *>(&u[k]);
#pragma unroll
          for (int e = 0; e < 8; e++)
            r[e] = k0 + k == 0 ? mul_rn(h2f(z[e]), sy[0]) : __fmaf_rn(h2f(z[e]), sy[k0 + k], r[e]);
        }
    }
    reinterpret_cast<float4 *>(out + i0)[0] = make_float4(r[0], r[1], r[2], r[3]);
    reinterpret_cast<float4 *>(out + i0)[1] = make_float4(r[4], r[5], r[6], r[7]);
  } else {
    for (int64_t i = i0; i < n; i++) {
      float r = mul_rn(h2f(Z[i]), sy[0]);
      for (int k = 1; k < nz; k++) r = __fmaf_rn(h2f(Z[k * ldz + i]), sy[k], r);
      out[i] = r;
    }
  }
}

}  // namespace f3r
