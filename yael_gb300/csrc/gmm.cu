// Gaussian mixture models with diagonal covariances (yael/gmm.c): EM learning
// seeded by k-means, posteriors p(component | vector), Fisher vectors.
//
// Two device passes carry every cost that grows with the number of vectors:
//   * posteriors: the squared Mahalanobis distance of every (vector,
//     component) pair in direct form, sum_l (x_l - mu_l)^2 / sigma_l, and the
//     reference's thresholded softmax of each vector's log densities on the
//     rows still in shared memory;
//   * moments: sum_i p_ij, sum_i p_ij x_il and sum_i p_ij x_il^2 for every
//     component and dimension (FP32 within each step of 32 vectors, pairs of
//     floats across steps, or FP64 where values are large, FP64 across vector
//     slices, summed in a fixed order: every result is reproducible), skipping
//     zero posteriors.
// Fisher vectors are formed on the device from those moments; the EM update of the
// k x d parameters and the empty-component splits are host code over them.  The posterior
// matrix (n x k) stays on the device between the passes of an EM iteration.
#include <cuda_runtime.h>
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "../../include/yael_gpu.h"
#include "common.cuh"

namespace yg {
namespace {

constexpr int GT = 32;                // tile edge of the count
constexpr float kNormTo0 = 16.636f;   // log(2^24) (yael/gmm.c:264)
constexpr float kMinSigma = 1e-10f;   // yael/gmm.c:111

// --- posteriors ------------------------------------------------------------
// One CTA computes the squared Mahalanobis distances of a tile of vectors to
// every component, keeps them in shared memory and turns each vector's row
// into posteriors there, so the n x k matrix is written once and never read
// back by this pass.  Bound by the FP32 pipe: three operations per (vector,
// component, dimension), a direct form whose differences do not cancel.  A
// thread holds VR vectors x 4 components (a warp 4 VR x 32, a CTA 16 VR x 128),
// so that 12 shared-memory wavefronts feed 192 operations; the operand slices
// of 32 dimensions are double-buffered with cp.async.  n = 100k, k = 256, d = 128:
// 0.62 ms + 0.28 ms for the 32 x 32 tiles and the separate softmax (whose FP64
// log densities and reciprocal held the narrow FP64 pipe) -> 0.48 ms
// (FP32 pipe alone: 0.27).
constexpr int MT = 512;                // threads: 4 x 4 warps of components x vectors
constexpr int MC = 128;                // components per pass of the tile
constexpr int ML = 32, MLD = ML + 4;   // dimensions per slice, row pitch (conflict-free float4)

// floats of dynamic shared memory: two operand buffers and the tile's rows
__host__ __device__ constexpr size_t maha_floats(int vr, int k) {
  return (size_t)2 * (16 * vr + 2 * MC) * MLD + (size_t)16 * vr * (k + 1);
}

__device__ __forceinline__ void cp_async(float *dst, const float *src, int bytes, bool ok) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(dst);
  if (bytes == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(src),
                 "r"(ok ? 16 : 0));
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(s), "l"(src),
                 "r"(ok ? 4 : 0));
}

// The log density logdet_j - 0.5 M + lg_j (yael/gmm.c:349-354) rounded to
// float, from base_hi + base_lo = logdet_j + lg_j: the sum's rounding error is
// recovered exactly (two-sum), so this is the FP64 sum rounded to float
// without the FP64 pipe.
__device__ __forceinline__ float log_density(float M, float hi, float lo) {
  const float m = -0.5f * M;
  const float s = __fadd_rn(hi, m);
  if (!(fabsf(s) <= 3.4e38f)) return s;  // infinite or NaN: no error term
  const float t = __fsub_rn(s, hi);
  const float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, t)), __fsub_rn(m, t));
  return __fadd_rn(s, __fadd_rn(e, lo));
}

// softmax_ref (yael/gmm.c:262-300) of one vector by one warp: x_j below
// max - 16.636 gives 0, the others exp(x_j - max), all divided by their sum.
// row: squared distances on entry; the posteriors go to out (may be row).
__device__ __forceinline__ void softmax_row(float *row, float *out, const float *__restrict__ hi,
                                            const float *__restrict__ lo, int k, int lane) {
  float mx = -1e30f;
  for (int j = lane; j < k; j += 32) {
    const float x = log_density(row[j], hi[j], lo[j]);
    row[j] = x;
    if (x > mx) mx = x;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  const float thr = mx - kNormTo0;
  float s = 0.f;
  for (int j = lane; j < k; j += 32) {
    const float x = row[j];
    const float e = x >= thr ? expf(x - mx) : 0.f;
    row[j] = e;
    s += e;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  const float inv = s != 0.f ? __frcp_rn(s) : 1.f;
  for (int j = lane; j < k; j += 32) {
    const float p = row[j] * inv;
    row[j] = p;
    out[j] = p;
  }
}

// FUSED: P gets the posteriors, nnz (if not null) the counts of positive
// ones per component; else P gets the squared distances (k too large for the
// tile's rows in shared memory; softmax_kernel follows).
// PAD: a last slice of fewer than ML dimensions, whose padding is not worked
// through (d = 100: 74 -> 69 us for 20k vectors, k = 100; the test costs others 2 to 8%).
template <int VR, bool FUSED, bool PAD>
__global__ void __launch_bounds__(MT, 1)
    posterior_kernel(const float *__restrict__ v, const float *__restrict__ mu,
                     const float *__restrict__ isig, const float *__restrict__ hi,
                     const float *__restrict__ lo, long n, int k, int d, float *__restrict__ P,
                     int *__restrict__ nnz) {
  constexpr int VT = 16 * VR;
  extern __shared__ __align__(16) float sm[];
  constexpr int BUF = (VT + 2 * MC) * MLD;
  float *rows = sm + 2 * BUF;  // [VT][k + 1]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int lc = lane & 7, lv = lane >> 3, wc = warp & 3, wv = warp >> 2;
  const long i0 = (long)blockIdx.x * VT;
  const int nl = (d + ML - 1) / ML, nc = (k + MC - 1) / MC, nit = nl * nc;
  const bool wide = (d & 3) == 0;

  auto stage = [&](int it) {  // operand slices of step it into buffer it & 1
    const int j0 = (it / nl) * MC, l0 = (it % nl) * ML;
    float *b = sm + (it & 1) * BUF;
    const int sh = wide ? 3 : 5;  // 8 copies of four floats or 32 of one per row
    for (int t = tid; t < (VT + 2 * MC) << sh; t += MT) {
      const int r = t >> sh, c = (t - (r << sh)) * (wide ? 4 : 1);
      const int l = l0 + c;
      const float *src;
      bool ok = l < d;
      if (r < VT) {
        ok = ok && i0 + r < n;
        src = ok ? v + (i0 + r) * d + l : v;
      } else {
        const int j = j0 + ((r - VT) & (MC - 1));
        ok = ok && j < k;
        const float *a = r < VT + MC ? mu : isig;
        src = ok ? a + (long)j * d + l : a;
      }
      cp_async(b + r * MLD + c, src, wide ? 16 : 4, ok);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  float acc[VR][4];
  stage(0);
  for (int it = 0; it < nit; it++) {
    if (it + 1 < nit) {
      stage(it + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    if (it % nl == 0) {
#pragma unroll
      for (int r = 0; r < VR; r++)
#pragma unroll
        for (int c = 0; c < 4; c++) acc[r][c] = 0.f;
    }
    const float *xs = sm + (it & 1) * BUF + (wv * 4 * VR + lv) * MLD;
    const float *ms = sm + (it & 1) * BUF + (VT + wc * 32 + lc) * MLD;
    const float *is = ms + MC * MLD;
    const int left = d - (it % nl) * ML;
#pragma unroll
    for (int l = 0; l < ML; l += 4) {
      if (PAD && l >= left) break;
      float4 x[VR];
#pragma unroll
      for (int r = 0; r < VR; r++)
        x[r] = *reinterpret_cast<const float4 *>(xs + 4 * r * MLD + l);
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const float4 m = *reinterpret_cast<const float4 *>(ms + 8 * c * MLD + l);
        const float4 s = *reinterpret_cast<const float4 *>(is + 8 * c * MLD + l);
#pragma unroll
        for (int r = 0; r < VR; r++) {
          float t = x[r].x - m.x;
          acc[r][c] = fmaf(t * t, s.x, acc[r][c]);
          t = x[r].y - m.y;
          acc[r][c] = fmaf(t * t, s.y, acc[r][c]);
          t = x[r].z - m.z;
          acc[r][c] = fmaf(t * t, s.z, acc[r][c]);
          t = x[r].w - m.w;
          acc[r][c] = fmaf(t * t, s.w, acc[r][c]);
        }
      }
    }
    if (it % nl == nl - 1) {
#pragma unroll
      for (int r = 0; r < VR; r++) {
        const int i = wv * 4 * VR + lv + 4 * r;
#pragma unroll
        for (int c = 0; c < 4; c++) {
          const int j = (it / nl) * MC + wc * 32 + lc + 8 * c;
          if (j < k) {
            if (FUSED)
              rows[(long)i * (k + 1) + j] = acc[r][c];
            else if (i0 + i < n)
              P[(i0 + i) * k + j] = acc[r][c];
          }
        }
      }
    }
    __syncthreads();
  }
  if constexpr (FUSED) {
    for (int i = warp; i < VT; i += MT / 32) {
      if (i0 + i >= n) break;
      softmax_row(rows + (long)i * (k + 1), P + (i0 + i) * k, hi, lo, k, lane);
    }
    if (!nnz) return;
    __syncthreads();
    const int nv = (int)min((long)VT, n - i0);
    for (int j = tid; j < k; j += MT) {
      int c = 0;
      for (int i = 0; i < nv; i++) c += rows[(long)i * (k + 1) + j] > 0.f ? 1 : 0;
      if (c) atomicAdd(nnz + j, c);
    }
  }
}

// one warp per vector, in place on its row of P (squared Mahalanobis
// distances on entry)
__global__ void softmax_kernel(float *__restrict__ P, const float *__restrict__ hi,
                               const float *__restrict__ lo, long n, int k) {
  const int lane = threadIdx.x & 31;
  const long i = (long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i >= n) return;  // whole warps leave together
  softmax_row(P + i * k, P + i * k, hi, lo, k, lane);
}

// --- moments ---------------------------------------------------------------
// part[z] = { S1[k][d], S2[k][d], S0[k] } of vector slice z: sum_i p_ij x_il,
// sum_i p_ij x_il^2 and sum_i p_ij over vectors [z*chunk, min(n, (z+1)*chunk)).
//
// A warp owns CPW components and DPL dimensions per lane, so a posterior is
// uniform over the warp and a (vector, components) pair whose posteriors are
// all zero is skipped by the whole warp: a thresholded softmax leaves few
// components per vector, and the pass then costs its reads.  (0 * x is only
// left out for finite x; a row with an infinity or a NaN is never skipped.)
// Dense posteriors are bound by the FP32 pipe: two packed multiply-adds per
// two dimensions and component.  Sums are FP32 within each step of 32 vectors
// and pairs of floats (two-sum, 2^-48) across steps: FP64 additions there held the
// FP64 pipe, 4 of its operations per 64 multiply-adds at 1/64 the rate.  Slices
// are summed in FP64 in a fixed order.  Against 64-bit moments the mean error
// is 0.77 to 1.00 of what FP64 sums across the steps gave (32 mixtures of 200 to
// 100k vectors, d = 16 to 128, k = 4 to 256): the steps' float sums set it.
// n = 100k, k = 256, d = 128: 1.25 ms -> 0.21 ms on average over ten EM iterations
// (all posteriors positive in the first, 0.5% of them from the third on).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float lo2(f32x2 a) { return __uint_as_float((unsigned)a); }
__device__ __forceinline__ float hi2(f32x2 a) { return __uint_as_float((unsigned)(a >> 32)); }
constexpr f32x2 kMinusOne2 = 0xbf800000bf800000ull;

// s + c += y: the rounding error of s + y is exact (two-sum) and goes to c, so
// the pair holds the sum to about 2^-48 (a Kahan sum would round y to
// float once more per step)
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) { return fma2(b, kMinusOne2, a); }
__device__ __forceinline__ void acc2(f32x2 &s, f32x2 &c, f32x2 y) {
  const f32x2 t = add2(s, y), b = sub2(t, s);
  c = add2(c, add2(sub2(s, sub2(t, b)), sub2(y, b)));
  s = t;
}
// A slice with a value that could overflow a float sum (an infinity or a NaN too)
// is summed again with two FP64 sums in a pair's registers, so that its sums are
// finite, infinite or NaN as FP64 sums are: of the low float in s, the high in c.
__device__ __forceinline__ double as_d(f32x2 a) { return __longlong_as_double((long long)a); }
__device__ __forceinline__ f32x2 d_as(double a) { return (f32x2)__double_as_longlong(a); }
__device__ __forceinline__ void to64(f32x2 &s, f32x2 &c) {
  const double a = (double)lo2(s) + (double)lo2(c), b = (double)hi2(s) + (double)hi2(c);
  s = d_as(a);
  c = d_as(b);
}
__device__ __forceinline__ void acc64(f32x2 &s, f32x2 &c, f32x2 y) {
  s = d_as(as_d(s) + (double)lo2(y));
  c = d_as(as_d(c) + (double)hi2(y));
}
// an infinity, a NaN or a value of 2^64 / h or more among the four.  2^34 for
// coordinates and 2^20 for posteriors: below them 2^31 products p x^2 add up to
// less than 2^119.
__device__ __forceinline__ bool big4(float4 x, float h) {
  const float a = x.x * h, b = x.y * h, c = x.z * h, d = x.w * h;
  const float z = 0.f * (a * a) + 0.f * (b * b) + 0.f * (c * c) + 0.f * (d * d);
  return z != z;
}
constexpr float kBigX = 1073741824.f, kBigP = 17592186044416.f;  // 2^30, 2^44

template <int NW, int DPL>
__global__ void __launch_bounds__(NW * 32, 16 / NW)
    moments_kernel(const float *__restrict__ P, const float *__restrict__ v, long n, int k, int d,
                   long chunk, double *__restrict__ part) {
  constexpr int CPW = 16 / DPL;     // components per warp
  constexpr int CT = NW * CPW;      // components per CTA
  constexpr int XW = 32 * DPL;      // dimensions per CTA
  constexpr int PLD = 2 * CT + 4;   // posteriors twice each (packed operands), padded
  constexpr int H = DPL / 2;        // packed pairs per lane
  constexpr int NT = NW * 32;
  constexpr int XQ = 32 * XW / 4 / NT, PQ = (32 * CT / 4 + NT - 1) / NT;  // float4 per thread
  constexpr bool PRE = NW == 16;    // one CTA per SM: the next step's loads fly meanwhile
  extern __shared__ __align__(16) float sm[];
  float(*xs)[32][XW] = reinterpret_cast<float(*)[32][XW]>(sm);
  float(*ps)[32][PLD] = reinterpret_cast<float(*)[32][PLD]>(sm + 2 * 32 * XW);
  __shared__ unsigned bad[3];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int l0 = blockIdx.x * XW, j0 = blockIdx.y * CT;
  const long ib = (long)blockIdx.z * chunk, ie = min(n, ib + chunk);
  const bool vx = (d & 3) == 0, vp = (k & 3) == 0;

  float4 rx[XQ], rp[PQ];
  auto load4 = [&](const float *base, long row, int w, int c, bool wide) {
    float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row >= ie) return r;
    const float *q = base + row * w + c;
    if (wide) {
      if (c < w) r = *reinterpret_cast<const float4 *>(q);
    } else {
      if (c < w) r.x = q[0];
      if (c + 1 < w) r.y = q[1];
      if (c + 2 < w) r.z = q[2];
      if (c + 3 < w) r.w = q[3];
    }
    return r;
  };
  auto gload = [&](long c0) {
#pragma unroll
    for (int q = 0; q < XQ; q++) {
      const int t = tid + q * NT, r = t / (XW / 4), c = (t % (XW / 4)) * 4;
      rx[q] = load4(v, c0 + r, d, l0 + c, vx);
    }
#pragma unroll
    for (int q = 0; q < PQ; q++) {
      const int t = tid + q * NT, r = t / (CT / 4), c = (t % (CT / 4)) * 4;
      if (r < 32) rp[q] = load4(P, c0 + r, k, j0 + c, vp);
    }
  };
  auto sstore = [&](int buf, int b3) {
#pragma unroll
    for (int q = 0; q < XQ; q++) {
      const int t = tid + q * NT, r = t / (XW / 4), c = (t % (XW / 4)) * 4;
      *reinterpret_cast<float4 *>(&xs[buf][r][c]) = rx[q];
      if (big4(rx[q], kBigX)) atomicOr(&bad[b3], 1u << r);
    }
#pragma unroll
    for (int q = 0; q < PQ; q++) {
      const int t = tid + q * NT, r = t / (CT / 4), c = (t % (CT / 4)) * 4;
      if (r < 32) {
        float4 *o = reinterpret_cast<float4 *>(&ps[buf][r][2 * c]);
        o[0] = make_float4(rp[q].x, rp[q].x, rp[q].y, rp[q].y);
        o[1] = make_float4(rp[q].z, rp[q].z, rp[q].w, rp[q].w);
      }
    }
  };

  f32x2 s1[CPW][H], c1[CPW][H], s2[CPW][H], c2[CPW][H];
  f32x2 s0[CPW / 2], c0s[CPW / 2];  // two components each
  // The sums of the slice; whether this warp met a value that is not for pairs
  // of floats (big4).  wide: FP64 sums in the pairs' registers (acc64).
  auto pass = [&](auto wide_) -> bool {
    constexpr bool wide = decltype(wide_)::value;
#pragma unroll
    for (int c = 0; c < CPW; c++) {
      s0[c / 2] = c0s[c / 2] = 0ull;
#pragma unroll
      for (int h = 0; h < H; h++) s1[c][h] = c1[c][h] = s2[c][h] = c2[c][h] = 0ull;
    }
    if (tid < 3) bad[tid] = 0u;
    __syncthreads();
    if (PRE) gload(ib);
    int step = 0;
    bool big = false;
    for (long i = ib; i < ie; i += 32, step++) {
      const int buf = step & 1, b3 = step % 3;
      if (!PRE) gload(i);
      sstore(buf, b3);
      __syncthreads();
      if (tid == 0) bad[(step + 2) % 3] = 0u;
      if (PRE && i + 32 < ie) gload(i + 32);
      // lane = vector: which vectors have a positive posterior here
      const float *prow = &ps[buf][0][2 * warp * CPW];
      bool any = false;
#pragma unroll
      for (int c = 0; c < CPW; c += 2) {
        const float4 p = *reinterpret_cast<const float4 *>(prow + lane * PLD + 2 * c);
        any = any || p.x != 0.f || p.z != 0.f;
        big = big || big4(p, kBigP);
        if (blockIdx.x == 0) {
          const f32x2 y = (f32x2)__float_as_uint(p.z) << 32 | __float_as_uint(p.x);
          if (wide) acc64(s0[c / 2], c0s[c / 2], y);
          else acc2(s0[c / 2], c0s[c / 2], y);
        }
      }
      unsigned m = __ballot_sync(0xffffffffu, any) | bad[b3];
      big = big || bad[b3];
      if (!m) continue;
      f32x2 f1[CPW][H], f2[CPW][H];
#pragma unroll
      for (int c = 0; c < CPW; c++)
#pragma unroll
        for (int h = 0; h < H; h++) f1[c][h] = f2[c][h] = 0ull;
      do {
        const int ii = __ffs(m) - 1;
        m &= m - 1;
        f32x2 x[H];
        if (H == 2) {
          const ulonglong2 t = *reinterpret_cast<const ulonglong2 *>(&xs[buf][ii][lane * DPL]);
          x[0] = t.x;
          x[H - 1] = t.y;
        } else {
          x[0] = *reinterpret_cast<const f32x2 *>(&xs[buf][ii][lane * DPL]);
        }
#pragma unroll
        for (int c = 0; c < CPW; c += 2) {
          const ulonglong2 p =
              *reinterpret_cast<const ulonglong2 *>(prow + ii * PLD + 2 * c);
#pragma unroll
          for (int h = 0; h < H; h++) {
            f1[c][h] = fma2(p.x, x[h], f1[c][h]);
            f1[c + 1][h] = fma2(p.y, x[h], f1[c + 1][h]);
            const f32x2 xx = mul2(x[h], x[h]);
            f2[c][h] = fma2(p.x, xx, f2[c][h]);
            f2[c + 1][h] = fma2(p.y, xx, f2[c + 1][h]);
          }
        }
      } while (m);
#pragma unroll
      for (int c = 0; c < CPW; c++)
#pragma unroll
        for (int h = 0; h < H; h++) {
          if (wide) {
            acc64(s1[c][h], c1[c][h], f1[c][h]);
            acc64(s2[c][h], c2[c][h], f2[c][h]);
          } else {
            acc2(s1[c][h], c1[c][h], f1[c][h]);
            acc2(s2[c][h], c2[c][h], f2[c][h]);
          }
        }
    }
    return big;
  };
  const bool wide = __syncthreads_or(pass(std::false_type()));
  if (wide) (void)pass(std::true_type());  // rare: the slice again

  double *out = part + (long)blockIdx.z * k * (2L * d + 1);
#pragma unroll
  for (int c = 0; c < CPW; c++) {
    const int j = j0 + warp * CPW + c;
    if (j >= k) break;
    if (blockIdx.x == 0) {
      if (!wide && !(c & 1)) to64(s0[c / 2], c0s[c / 2]);
      double t = as_d(c & 1 ? c0s[c / 2] : s0[c / 2]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (lane == 0) out[2L * k * d + j] = t;
    }
#pragma unroll
    for (int h = 0; h < H; h++) {
      const int l = l0 + lane * DPL + 2 * h;
      const long o = (long)j * d + l;
      if (!wide) {
        to64(s1[c][h], c1[c][h]);
        to64(s2[c][h], c2[c][h]);
      }
      if (l < d) {
        out[o] = as_d(s1[c][h]);
        out[(long)k * d + o] = as_d(s2[c][h]);
      }
      if (l + 1 < d) {
        out[o + 1] = as_d(c1[c][h]);
        out[(long)k * d + o + 1] = as_d(c2[c][h]);
      }
    }
  }
}

// out[t] = sum over slices z (in order) of part[z * m + t]
__global__ void sum_slices_kernel(const double *__restrict__ part, int nz, long m,
                                  double *__restrict__ out) {
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= m) return;
  double s = 0;
#pragma unroll 8
  for (int z = 0; z < nz; z++) s += part[(long)z * m + t];
  out[t] = s;
}

// --- parameters --------------------------------------------------------------
// From a mixture's (w, mu, sigma): 1 / sigma, and the constant terms of the log
// density of each component, log det + log w (yael/gmm.c:311-330, the
// determinant accumulated in float as there), in two floats.  A warp per
// component: the logarithms by its lanes, their sum in order.
__global__ void params_kernel(const float *__restrict__ w, const float *__restrict__ sigma, int k,
                              int d, float det0, int use_w, float *__restrict__ isig,
                              float *__restrict__ hi, float *__restrict__ lo) {
  const int lane = threadIdx.x & 31;
  const int j = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (j >= k) return;  // whole warps leave together
  float det = det0;
  for (int l0 = 0; l0 < d; l0 += 32) {
    const int l = l0 + lane;
    double h = 0.0;
    if (l < d) {
      const double sg = sigma[(long)j * d + l];
      isig[(long)j * d + l] = (float)(1.0 / sg);
      h = 0.5 * log(sg);
    }
    const int m = min(32, d - l0);
    for (int s = 0; s < m; s++) det = (float)((double)det - __shfl_sync(0xffffffffu, h, s));
  }
  if (lane == 0) {
    const double base = (double)det + (use_w ? (double)(float)log((double)w[j]) : 0.0);
    const float h = (float)base;
    hi[j] = h;
    lo[j] = isfinite(base) ? (float)(base - (double)h) : 0.f;
  }
}

// --- Fisher vectors ------------------------------------------------------------
// gmm_fisher_from_posteriors (yael/gmm.c:527-725) from the FP64 moments
// (S1[k][d], S2[k][d], S0[k]), each operation rounded on its own as in C.  On the
// device so that one image's vector comes back as floats: moving the moments
// to the host and dividing there took longer than all the passes of 2,000
// descriptors.  Thread t < k*d: dimension t % d of component t / d; the parts
// that sum over dimensions (GMM_FLAGS_1SIGMA) go a component per thread.
__device__ __forceinline__ double dev2_of(double mu, double s0, double s1, double s2) {
  return __dadd_rn(__dsub_rn(s2, __dmul_rn(__dmul_rn(2.0, mu), s1)), __dmul_rn(__dmul_rn(mu, mu), s0));
}

__global__ void fisher_kernel(const double *__restrict__ sum, const float *__restrict__ w,
                              const float *__restrict__ mu, const float *__restrict__ sigma,
                              long n, int k, int d, int flags, float *__restrict__ out) {
  const long kd = (long)k * d, t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const double *s1 = sum, *s2 = sum + kd, *s0 = sum + 2 * kd;
  const bool norm = !(flags & YAEL_GMM_FLAGS_NO_NORM);
  if (flags & YAEL_GMM_FLAGS_W) {
    if (t >= 1 && t < k) {
      const double accu = __dsub_rn(s0[t] / w[t], s0[0] / w[0]);
      const double f = __dmul_rn((double)n, __dadd_rn(1.0 / w[t], 1.0 / w[0]));
      out[t - 1] = (float)(accu / sqrt(f));
    }
    out += k - 1;
  }
  if (t >= kd) return;
  const int j = (int)(t / d);
  const double m = mu[t], sg = sigma[t], wj = w[j];
  if (flags & YAEL_GMM_FLAGS_MU) {
    double x = __dsub_rn(s1[t], __dmul_rn(m, s0[j])) / sg;
    if (norm) {
      const double nf = sqrt(__dmul_rn((double)n, wj) / sg);
      if (nf > 0) x /= nf;
    }
    out[t] = (float)x;
    out += kd;
  }
  if (flags & YAEL_GMM_FLAGS_1SIGMA) {
    if (t != (long)j * d) return;
    const bool each = flags & YAEL_GMM_FLAGS_SIGMA;
    float *o = out + (each ? (long)j * (d + 1) : j);
    double accu2 = 0;
    for (int l = 0; l < d; l++) {
      const long u = t + l;
      const double su = sigma[u];
      const double accu =
          __dsub_rn(dev2_of(mu[u], s0[j], s1[u], s2[u]) / su, s0[j]) / sqrt(su);
      if (each)
        *o++ = (float)(accu / sqrt(norm ? __dmul_rn((double)(2 * n), wj) / su : 1.0));
      accu2 = __dadd_rn(accu2, accu);
    }
    *o = (float)(accu2 / sqrt(norm ? __dmul_rn((double)(2 * d * n), wj) / sg : 1.0));
  } else if (flags & YAEL_GMM_FLAGS_SIGMA) {
    const double accu = __dsub_rn(dev2_of(m, s0[j], s1[t], s2[t]), __dmul_rn(s0[j], sg));
    const double f =
        norm ? 1 / __dmul_rn(sg, sqrt(__dmul_rn((double)(2 * n), wj))) : pow(sg, -1.5);
    out[t] = (float)__dmul_rn(accu, f);
  }
}

// nnz[j] += number of vectors of slice y with P[i*k + j] > 0.  Block 32 x 8:
// thread (tx, ty) counts component j0 + tx over vectors ty, ty + 8, ...
__global__ void nnz_kernel(const float *__restrict__ P, long n, int k, long chunk,
                           int *__restrict__ nnz) {
  __shared__ int red[8][GT];
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int j = blockIdx.x * GT + tx;
  const long ib = (long)blockIdx.y * chunk, ie = min(n, ib + chunk);
  int c = 0;
  if (j < k)
    for (long i = ib + ty; i < ie; i += 8) c += P[i * k + j] > 0.f ? 1 : 0;
  red[ty][tx] = c;
  __syncthreads();
  if (ty == 0 && j < k) {
    int t = 0;
    for (int q = 0; q < 8; q++) t += red[q][tx];
    if (t) atomicAdd(nnz + j, t);
  }
}

// the split of gmm_handle_empty (yael/gmm.c:404-411): vectors with
// P[., j2] > 0 and v[., sd] < thr move their posterior from j2 to j
__global__ void transfer_kernel(float *__restrict__ P, const float *__restrict__ v, long n,
                                int k, int d, int j, int j2, int sd, float thr,
                                int *__restrict__ moved) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  int c = 0;
  if (i < n) {
    const float q = P[i * k + j2];
    if (q > 0.f && v[i * d + sd] < thr) {
      P[i * k + j] = q;
      P[i * k + j2] = 0.f;
      c = 1;
    }
  }
  c = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(moved, c);
}

[[noreturn]] void die(const char *where) { fatal_last(where); }

void ok(const char *where, cudaError_t e) {
  if (e != cudaSuccess) {
    set_error(E_CUDA, "%s", cudaGetErrorString(e));
    die(where);
  }
}

void launched(const char *where) {
  count_launch();
  ok(where, cudaGetLastError());
}

// The moments of a posterior matrix against a set of vectors, as FP64, in
// pinned memory of the context: s0[j] = sum_i p_ij, s1[j*d + l] = sum_i p_ij x_il,
// s2[j*d + l] = sum_i p_ij x_il^2
struct Moments {
  const double *s0, *s1, *s2;
};

// A device array of a call: workspace of the calling thread up to kKeepBytes
// (one image's descriptors: allocating and freeing ten arrays took 0.4 of a
// 0.6 ms call), an allocation of the call's own above (given back at its end).
constexpr size_t kKeepBytes = (size_t)32 << 20;
enum GmmSlot : int {
  GM_V = 260, GM_P, GM_PRM, GM_ISIG, GM_HI, GM_LO, GM_PART, GM_SUM, GM_NNZ, GM_MOVED, GM_OUT,
};
template <typename T, int SLOT>
struct GmmArray {
  T *p = nullptr;
  DevArray<T> own;
  T *get(Ctx *ctx, const char *where, long want) {
    const size_t bytes = sizeof(T) * (size_t)(want > 1 ? want : 1);
    if (bytes > kKeepBytes) {
      p = own.get(where, want);
    } else {
      void *q = nullptr;
      if (ctx->ws.get(SLOT, bytes, &q) != OK) die(where);
      p = static_cast<T *>(q);
    }
    return p;
  }
};
// pinned buffers: parameters and small vectors on their way up, moments down
enum GmmPinned : int { GP_PRM = 8, GP_V, GP_MOMENTS };

// device state of one call: vectors, posteriors, parameters, moments
struct GmmDev {
  const char *where;
  Ctx *ctx = nullptr;
  long n = 0;
  int d = 0, k = 0;
  GmmArray<float, GM_V> v;
  GmmArray<float, GM_P> P;
  GmmArray<float, GM_PRM> prm;  // mu[k][d], sigma[k][d], w[k]
  GmmArray<float, GM_ISIG> isig;
  GmmArray<float, GM_HI> dhi;
  GmmArray<float, GM_LO> dlo;
  GmmArray<double, GM_PART> part;
  GmmArray<double, GM_SUM> sum;
  GmmArray<int, GM_NNZ> nnz;
  GmmArray<int, GM_MOVED> moved;
  GmmArray<float, GM_OUT> fv;

  GmmDev(const char *w, long n_, int d_, int k_) : where(w), n(n_), d(d_), k(k_) {
    if (ctx_get(&ctx) != OK) die(where);
  }
  void sync() { ok(where, cudaStreamSynchronize(ctx->stream)); }
  void *pinned(int slot, size_t bytes) {
    void *h = nullptr;
    if (ctx->pinned.get(slot, bytes, &h) != OK) die(where);
    return h;
  }
  void upload_v(const float *hv) {
    const size_t bytes = sizeof(float) * (size_t)(n * d);
    if (copy_to_device(ctx, ctx->stream, GP_V, v.get(ctx, where, n * d), hv, bytes) != OK)
      die(where);
  }
  void upload_P(const float *hp) {
    ok(where, cudaMemcpyAsync(P.get(ctx, where, n * k), hp, sizeof(float) * (size_t)(n * k),
                              cudaMemcpyHostToDevice, ctx->stream));
  }
  void download_P(float *hp) {
    if (copy_to_host(ctx->stream, hp, P.p, sizeof(float) * (size_t)(n * k)) != OK) die(where);
  }

  // the mixture on the device (one copy from pinned memory; the caller
  // synchronises before the next)
  void upload_params(const gmm_t *g) {
    const size_t kd = (size_t)k * d, m = 2 * kd + k;
    float *h = static_cast<float *>(pinned(GP_PRM, sizeof(float) * m));
    memcpy(h, g->mu, sizeof(float) * kd);
    memcpy(h + kd, g->sigma, sizeof(float) * kd);
    memcpy(h + 2 * kd, g->w, sizeof(float) * k);
    ok(where, cudaMemcpyAsync(prm.get(ctx, where, (long)m), h, sizeof(float) * m,
                              cudaMemcpyHostToDevice, ctx->stream));
  }
  const float *mu_dev() const { return prm.p; }
  const float *sigma_dev() const { return prm.p + (size_t)k * d; }
  const float *w_dev() const { return prm.p + 2 * (size_t)k * d; }

  // P = p(component | vector) for the mixture (w, mu, sigma): gmm_compute_p
  // (yael/gmm.c:305-362); flags & GMM_FLAGS_W adds log w_j.  count: also leave
  // the number of vectors with a positive posterior per component in nnz.
  void posteriors(const gmm_t *g, int flags, bool count = false) {
    const long kd = (long)k * d;
    cudaStream_t st = ctx->stream;
    upload_params(g);
    isig.get(ctx, where, kd);
    dhi.get(ctx, where, k);
    dlo.get(ctx, where, k);
    params_kernel<<<(unsigned)((k + 3) / 4), 128, 0, st>>>(
        w_dev(), sigma_dev(), k, d, (float)(-d / 2.0 * log(2 * M_PI)),
        (flags & YAEL_GMM_FLAGS_W) != 0, isig.p, dhi.p, dlo.p);
    launched(where);
    P.get(ctx, where, n * k);
    if (count) ok(where, cudaMemsetAsync(nnz.get(ctx, where, k), 0, sizeof(int) * k, st));
    int *cnt = count ? nnz.p : nullptr;
    // The largest tile of vectors whose rows fit in shared memory and that
    // still gives every SM a CTA; k above about 2,300 fits none.
    const long sms = ctx->num_sms;
    if (fits(4) && n > 32 * sms)
      launch_posteriors<4, true>(cnt);
    else if (fits(2) && n > 16 * sms)
      launch_posteriors<2, true>(cnt);
    else if (fits(1))
      launch_posteriors<1, true>(cnt);
    else {
      launch_posteriors<4, false>(nullptr);
      softmax_kernel<<<(unsigned)((n + 7) / 8), 256, 0, st>>>(P.p, dhi.p, dlo.p, n, k);
      launched(where);
      if (count) count_nonzeros();
    }
  }

  bool fits(int vr) const { return maha_floats(vr, k) * sizeof(float) <= ctx->smem_optin; }

  template <int VR, bool FUSED>
  void launch_posteriors(int *cnt) {
    const size_t smem = maha_floats(VR, FUSED ? k : 0) * sizeof(float);
    const auto kern = d % ML ? posterior_kernel<VR, FUSED, true> : posterior_kernel<VR, FUSED, false>;
    if (ensure_smem((const void *)kern, smem) != OK) die(where);
    kern<<<(unsigned)((n + 16 * VR - 1) / (16 * VR)), MT, smem,
                                  ctx->stream>>>(v.p, mu_dev(), isig.p, dhi.p, dlo.p, n, k, d, P.p,
                                                 cnt);
    launched(where);
  }

  void count_nonzeros() {
    const long ny = std::min<long>(std::max<long>(1, (n + 4095) / 4096), 4096);
    const long chunk = (n + ny - 1) / ny;
    nnz_kernel<<<dim3((unsigned)((k + GT - 1) / GT), (unsigned)ny), dim3(GT, 8), 0,
                 ctx->stream>>>(P.p, n, k, chunk, nnz.p);
    launched(where);
  }

  // number of vectors with a positive posterior, per component (the counts of
  // the last posteriors(..., count = true))
  std::vector<int> nonzeros() {
    std::vector<int> h((size_t)k);
    ok(where, cudaMemcpyAsync(h.data(), nnz.p, sizeof(int) * k, cudaMemcpyDeviceToHost,
                              ctx->stream));
    sync();
    return h;
  }

  int transfer(int j, int j2, int sd, float thr) {
    cudaStream_t st = ctx->stream;
    ok(where, cudaMemsetAsync(moved.get(ctx, where, 1), 0, sizeof(int), st));
    transfer_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(P.p, v.p, n, k, d, j, j2, sd,
                                                                thr, moved.p);
    launched(where);
    int h = 0;
    ok(where, cudaMemcpyAsync(&h, moved.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    sync();
    return h;
  }

  template <int NW, int DPL>
  void launch_moments() {
    constexpr int CT = NW * 16 / DPL, XW = 32 * DPL;
    const long gx = (d + XW - 1) / XW, gy = (k + CT - 1) / CT;
    // one wave of resident CTAs, slices of at least two steps
    const long want = std::max(1L, ctx->num_sms * (16L / NW) / (gx * gy));
    const long steps = (n + 31) / 32;
    const long nz = std::max(1L, std::min(want, steps / 2));
    const long chunk = (steps + nz - 1) / nz * 32;
    const long m = (long)k * (2L * d + 1);
    const long used = (n + chunk - 1) / chunk;
    part.get(ctx, where, used * m);
    const size_t smem = sizeof(float) * 2 * 32 * (XW + 2 * CT + 4);
    if (ensure_smem((const void *)moments_kernel<NW, DPL>, smem) != OK) die(where);
    moments_kernel<NW, DPL><<<dim3((unsigned)gx, (unsigned)gy, (unsigned)used), NW * 32, smem,
                              ctx->stream>>>(P.p, v.p, n, k, d, chunk, part.p);
    launched(where);
    sum_slices_kernel<<<(unsigned)((m + 255) / 256), 256, 0, ctx->stream>>>(
        part.p, (int)used, m, sum.get(ctx, where, m));
    launched(where);
  }

  // the moments of P against v, in sum (S1, S2, S0)
  void moments_dev() {
    if (n == 0) {
      const size_t m = (size_t)k * (2 * (size_t)d + 1);
      ok(where, cudaMemsetAsync(sum.get(ctx, where, (long)m), 0, sizeof(double) * m, ctx->stream));
      return;
    }
    // Dimensions per lane by d.  16 warps to a CTA (fewer passes over the
    // vectors) where k gives the warps components of their own and n gives
    // every SM some steps; else 4-warp CTAs, four to an SM.  Both sums' passes in
    // us, 4-warp and 16-warp CTAs, dense posteriors, d = 64 and 128, k = 256: n = 500
    // 26 / 44 and 23 / 40; 2,000 37 / 52 and 42 / 50; 5,000 50 / 56 and 58 / 60;
    // 9,000 64 / 64 and 75 / 79; 20,000 93 / 93 and 130 / 126; 100,000 301 / 284 and
    // 549 / 484 (2% of them positive: 158 / 146 and 239 / 191).  k = 32, d = 128:
    // 121 / 118 at 100,000.
    const bool many = n >= 64L * ctx->num_sms;
    if (d > 64) {
      if (k > 32 && many) launch_moments<16, 4>(); else launch_moments<4, 4>();
    } else {
      if (k > 64 && many) launch_moments<16, 2>(); else launch_moments<4, 2>();
    }
  }

  Moments moments() {
    moments_dev();
    const size_t kd = (size_t)k * d, bytes = sizeof(double) * (2 * kd + k);
    double *h = static_cast<double *>(pinned(GP_MOMENTS, bytes));
    ok(where, cudaMemcpyAsync(h, sum.p, bytes, cudaMemcpyDeviceToHost, ctx->stream));
    sync();
    return Moments{h + 2 * kd, h, h + kd};
  }

  // the Fisher vector of P (or of no vectors) under the mixture in prm
  void fisher(int flags, float *out) {
    const long m = (long)gmm_len(flags);
    moments_dev();
    if (m == 0) {
      sync();
      return;
    }
    const long t = std::max((long)k * d, (long)k);
    fisher_kernel<<<(unsigned)((t + 127) / 128), 128, 0, ctx->stream>>>(
        sum.p, w_dev(), mu_dev(), sigma_dev(), n, k, d, flags, fv.get(ctx, where, m));
    launched(where);
    if (copy_to_host(ctx->stream, out, fv.p, sizeof(float) * (size_t)m) != OK) die(where);
  }
  size_t gmm_len(int flags) const {
    const gmm_t g{d, k, nullptr, nullptr, nullptr};
    return gmm_fisher_sizeof(&g, flags);
  }
};

gmm_t *gmm_alloc(int d, int k) {
  gmm_t *g = (gmm_t *)malloc(sizeof(gmm_t));
  g->d = d;
  g->k = k;
  g->w = (float *)malloc(sizeof(float) * (size_t)(k > 0 ? k : 1));
  g->mu = (float *)malloc(sizeof(float) * (size_t)((long)k * d + 1));
  g->sigma = (float *)malloc(sizeof(float) * (size_t)((long)k * d + 1));
  return g;
}

void print_fvec(const float *v, int n) {  // fvec_print (yael/vector.c:1587-1594)
  printf("[");
  for (int i = 0; i < n; i++) printf("%g ", v[i]);
  printf("]\n");
}

// gmm_handle_empty (yael/gmm.c:366-433): each component without any positive
// posterior takes, from the next component in steps of 1000003 (mod k) that
// has some and holds at least n / k vectors, the vectors below that
// component's mean along its dimension of largest variance
void handle_empty(GmmDev &dev, const gmm_t *g) {
  const long n = dev.n;
  const int k = dev.k, d = dev.d;
  const std::vector<int> nnz = dev.nonzeros();
  long nz = 0;
  for (int j = 0; j < k; j++) nz += n - nnz[j];
  printf("nb of 0 probabilities: %ld / (%ld*%ld) = %.1f %%\n", nz, (long)k, n,
         nz * 100.0 / ((double)k * n));
  // the reference's w[j] (a float sum of non-negative posteriors) is positive
  // exactly when the component has a positive posterior; -1 after a split
  std::vector<int> state((size_t)k);
  for (int j = 0; j < k; j++) state[j] = nnz[j] > 0 ? 1 : 0;
  const int bigprime = 1000003;
  for (int j = 0; j < k; j++) {
    if (state[j] != 0) continue;
    printf("center %d is empty....", j);
    fflush(stdout);
    int j2 = j, tries = 0;
    for (;;) {
      int i;
      for (i = 0; i < k; i++) {
        j2 = (int)(((long)j2 + bigprime) % k);
        if (state[j2] > 0) break;
      }
      if (i == k || ++tries > k) {
        set_error(E_ARG, "gmm_learn: could not find a component to split");
        die("gmm_learn");
      }
      printf("try share with cent %d...", j2);
      fflush(stdout);
      // a component is split once and never receives: its count is still nnz
      if (nnz[j2] < n / k) {
        printf("has too few pts (%d)...", nnz[j2]);
        fflush(stdout);
        continue;
      }
      break;
    }
    const float *sj2 = g->sigma + (long)d * j2;
    int sd = 0;  // fvec_arg_max: first maximum
    for (int l = 1; l < d; l++)
      if (sj2[l] > sj2[sd]) sd = l;
    const int nt = dev.transfer(j, j2, sd, g->mu[(long)j2 * d + sd]);
    printf("split %d at dim %d (variance %g, transferred %d/%d pts)\n", j2, sd, sj2[sd], nt,
           nnz[j2]);
    if (nt == nnz[j2] || nt == 0) printf("  still not balanced !!! (expect crash)\n");
    state[j2] = -1;
  }
}

// gmm_compute_params (yael/gmm.c:114-199) from the moments of the posteriors
void compute_params(GmmDev &dev, gmm_t *g, int flags) {
  const int k = dev.k, d = dev.d;
  const Moments m = dev.moments();
  const std::vector<float> mu_old(g->mu, g->mu + (long)k * d);
  for (int j = 0; j < k; j++) {
    g->w[j] = (float)m.s0[j];
    for (int l = 0; l < d; l++) {
      const size_t t = (size_t)j * d + l;
      const double mo = mu_old[t];
      g->mu[t] = (float)m.s1[t];
      // sum_i p_ij (x_il - mu_old_jl)^2, expanded around the previous means
      g->sigma[t] = (float)(m.s2[t] - 2.0 * mo * m.s1[t] + mo * mo * m.s0[j]);
    }
  }
  if (flags & YAEL_GMM_FLAGS_1SIGMA) {
    for (int j = 0; j < k; j++) {
      float *sj = g->sigma + (long)j * d;
      double s = 0;
      for (int l = 0; l < d; l++) s += sj[l];
      const float var = (float)(s / d);
      for (int l = 0; l < d; l++) sj[l] = var;
    }
  }
  long nz = 0;
  for (long t = 0; t < (long)k * d; t++)
    if (g->sigma[t] < kMinSigma) {
      g->sigma[t] = kMinSigma;
      nz++;
    }
  if (nz) printf("WARN %ld sigma diagonals are too small (set to %g)\n", nz, kMinSigma);
  double msum = 0;
  for (long t = 0; t < (long)k * d; t++) msum += g->mu[t];
  if (!isfinite(msum)) {
    set_error(E_ARG, "gmm_learn: non-finite means");
    die("gmm_learn");
  }
  for (int j = 0; j < k; j++) {  // fvec_div_by: times 1 / w in double
    const double inv = 1.0 / g->w[j];
    for (int l = 0; l < d; l++) {
      g->mu[(long)j * d + l] = (float)(g->mu[(long)j * d + l] * inv);
      g->sigma[(long)j * d + l] = (float)(g->sigma[(long)j * d + l] * inv);
    }
  }
  double wn = 0;  // fvec_normalize(w, k, 1)
  for (int j = 0; j < k; j++) wn += fabs((double)g->w[j]);
  for (int j = 0; j < k; j++) g->w[j] = (float)(g->w[j] * (1.0 / wn));
  printf("w = ");
  print_fvec(g->w, k);
  double ss = 0;
  for (int j = 0; j < k; j++) ss += (double)g->w[j] * g->w[j];
  printf(" imfac = %.3f\n", k * ss);
}

}  // namespace
}  // namespace yg

using namespace yg;

extern "C" {

void gmm_delete(gmm_t *g) {
  free(g->w);
  free(g->mu);
  free(g->sigma);
  free(g);
}

gmm_t *gmm_learn(int di, int ni, int ki, int niter, const float *v, int nt, int seed, int nredo,
                 int flags) {
  const long d = di, k = ki, n = ni;
  niter = niter == 0 ? 10000 : niter;
  gmm_t *g = gmm_alloc(di, ki);
  // initialisation: k-means, weights 1 / k, one variance for every diagonal
  std::vector<int> nassign((size_t)(k > 0 ? k : 1));
  std::vector<float> dis((size_t)(n > 0 ? n : 1));
  kmeans(di, ni, ki, niter, v, nt, seed, nredo, g->mu, dis.data(), nullptr, nassign.data());
  fflush(stderr);
  fprintf(stderr, "assign = ");
  fflush(stderr);
  printf("[");
  for (long j = 0; j < k; j++) printf("%d ", nassign[j]);
  printf("]\n");
  fprintf(stderr, "\n");
  for (long j = 0; j < k; j++) g->w[j] = (float)(1.0 / k);
  double sig = 0;
  for (long i = 0; i < n; i++) sig += dis[i];
  sig /= n;
  printf("sigma at initialization = %.3f\n", sig);
  for (long t = 0; t < k * d; t++) g->sigma[t] = (float)sig;
  fprintf(stdout, "<><><><> GMM  <><><><><>\n");
  if (flags & YAEL_GMM_FLAGS_PURE_KMEANS) niter = 0;
  if (niter > 0 && n > 0) {
    GmmDev dev("gmm_learn", n, di, ki);
    dev.upload_v(v);
    double key = 666, old_key;
    for (int iter = 1; iter <= niter; iter++) {
      dev.posteriors(g, flags, true);
      fflush(stdout);
      handle_empty(dev, g);
      compute_params(dev, g, flags);
      fflush(stdout);
      old_key = key;
      key = 0;
      for (long t = 0; t < k * d; t++) key += g->mu[t];
      printf("keys %5d: %.6f -> %.6f\n", iter, old_key, key);
      fflush(stdout);
      if (key == old_key) break;
    }
  }
  fprintf(stderr, "\n");
  return g;
}

void gmm_compute_p(int n, const float *v, const gmm_t *g, float *p, int flags) {
  if (n == 0) return;
  GmmDev dev("gmm_compute_p", n, g->d, g->k);
  dev.upload_v(v);
  dev.posteriors(g, flags);
  dev.download_P(p);
}

void gmm_compute_p_thread(int n, const float *v, const gmm_t *g, float *p, int flags,
                          int n_thread) {
  (void)n_thread;
  gmm_compute_p(n, v, g, p, flags);
}

size_t gmm_fisher_sizeof(const gmm_t *g, int flags) {
  int sz = 0;
  if (flags & YAEL_GMM_FLAGS_W) sz += g->k - 1;
  if (flags & YAEL_GMM_FLAGS_MU) sz += g->d * g->k;
  if (flags & YAEL_GMM_FLAGS_1SIGMA) sz += g->k;
  if (flags & YAEL_GMM_FLAGS_SIGMA) sz += g->d * g->k;
  return sz;
}

void gmm_fisher(int n, const float *v, const gmm_t *g, int flags, float *dp_dlambda) {
  GmmDev dev("gmm_fisher", n, g->d, g->k);
  if (n > 0) {
    dev.upload_v(v);
    dev.posteriors(g, flags | YAEL_GMM_FLAGS_W);
  } else {
    dev.upload_params(g);
  }
  dev.fisher(flags, dp_dlambda);
}

void gmm_fisher_from_posteriors(int n, const float *v, const gmm_t *g, int flags,
                                const float *p, float *dp_dlambda) {
  GmmDev dev("gmm_fisher_from_posteriors", n, g->d, g->k);
  if (n > 0) {
    dev.upload_v(v);
    dev.upload_P(p);
  }
  dev.upload_params(g);
  dev.fisher(flags, dp_dlambda);
}

void gmm_fisher_spatial(int N, int K, int D, const float *Q, const float *sgmm, const float *ll,
                        float *sdesc) {
  // ll is D x N (coordinate d of vector i at ll[d * N + i]): transposed to
  // the vector-major layout of the moments pass
  std::vector<float> llt((size_t)N * D + 1);
  for (long i = 0; i < N; i++)
    for (long c = 0; c < D; c++) llt[i * D + c] = ll[c * N + i];
  GmmDev dev("gmm_fisher_spatial", N, D, K);
  if (N > 0) {
    dev.upload_v(llt.data());
    dev.upload_P(Q);
  }
  const Moments m = dev.moments();
  const float *mm = sgmm, *S = sgmm + D;
  float *d_mm = sdesc, *d_S = sdesc + (long)K * D;
  for (long c = 0; c < D; c++)
    for (long j = 0; j < K; j++) {
      const double qs = m.s0[j] / N, ql = m.s1[j * D + c] / N, ql2 = m.s2[j * D + c] / N;
      d_mm[c + j * D] = (float)(ql - qs * mm[c]);
      d_S[c + j * D] = (float)(-ql2 + 2 * ql * mm[c] + qs * ((double)S[c] - (double)mm[c] * mm[c]));
    }
}

void gmm_print(const gmm_t *g) {
  printf("gmm (%d gaussians in %d dim)=[\n", g->k, g->d);
  for (int i = 0; i < g->k; i++) {
    printf("   w=%g, mu=[", g->w[i]);
    for (int j = 0; j < g->d; j++) printf("%g ", g->mu[(long)i * g->d + j]);
    printf("], sigma=diag([");
    for (int j = 0; j < g->d; j++) printf("%g ", g->sigma[(long)i * g->d + j]);
    printf("])\n");
  }
  printf("]\n");
}

// gmm_write / gmm_read (yael/gmm.c:810-850): d, k, w, mu, sigma as raw int32
// and float32; an I/O error prints and aborts
static void write_or_abort(const void *a, size_t sz, size_t n, FILE *f) {
  if (fwrite(a, sz, n, f) != n) {
    perror("gmm_write");
    abort();
  }
}

static void read_or_abort(void *a, size_t sz, size_t n, FILE *f) {
  if (fread(a, sz, n, f) != n) {
    perror("gmm_read");
    abort();
  }
}

void gmm_write(const gmm_t *g, FILE *f) {
  write_or_abort(&g->d, sizeof(int), 1, f);
  write_or_abort(&g->k, sizeof(int), 1, f);
  write_or_abort(g->w, sizeof(float), (size_t)g->k, f);
  write_or_abort(g->mu, sizeof(float), (size_t)g->k * g->d, f);
  write_or_abort(g->sigma, sizeof(float), (size_t)g->k * g->d, f);
}

gmm_t *gmm_read(FILE *f) {
  int d, k;
  read_or_abort(&d, sizeof(int), 1, f);
  read_or_abort(&k, sizeof(int), 1, f);
  gmm_t *g = gmm_alloc(d, k);
  read_or_abort(g->w, sizeof(float), (size_t)k, f);
  read_or_abort(g->mu, sizeof(float), (size_t)k * d, f);
  read_or_abort(g->sigma, sizeof(float), (size_t)k * d, f);
  return g;
}

}  // extern "C"
