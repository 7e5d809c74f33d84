// Row preparation: norms, exact-class flags, bf16 packing (see prep.cuh).
#include "prep.cuh"

#include <algorithm>

#include "scan.cuh"

namespace yg {

namespace {
constexpr int PW = 8;  // warps per block

// 16-bit operand encoding of the tensor-core passes: bf16 (F16 = false) or
// IEEE fp16 (F16 = true), both round to nearest even
template <bool F16>
__device__ __forceinline__ uint16_t to16(float v) {
  if (F16) return __half_as_ushort(__float2half_rn(v));
  return __bfloat16_as_ushort(__float2bfloat16_rn(v));
}
template <bool F16>
__device__ __forceinline__ float from16(uint16_t h) {
  if (F16) return __half2float(__ushort_as_half(h));
  return __bfloat162float(__ushort_as_bfloat16(h));
}

// the rounding error of the packed value of v: bf16 shares float's exponent
// range, so bf16(scale * v) = scale * bf16(v) for the power-of-two scales
// used (1, -2); fp16 does not (overflow above 65504, subnormals below 2^-14),
// so its error is taken from the packed value itself (an overflow gives an
// infinite error, which rejects the row's every result)
// (inv = 1 / scale, exact for these scales)
template <bool F16>
__device__ __forceinline__ float pack_err(float v, float inv, uint16_t packed) {
  if (F16) return v - from16<true>(packed) * inv;
  return v - __bfloat162float(__float2bfloat16_rn(v));
}

// the translation row of row r (null without one)
__device__ __forceinline__ const float *row_mu(const RowShift &sh, long r, int d) {
  if (!sh.mu) return nullptr;
  const long i = sh.row_inst ? (long)sh.row_inst[r] : r / sh.rows_per_inst;
  return sh.mu + i * d;
}

__device__ __forceinline__ float4 sub4(float4 a, float4 b) {
  return make_float4(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z),
                     __fsub_rn(a.w, b.w));
}

// the float norm as three 16-bit parts (11 + 11 + 11 or 8 + 8 + 8 significant
// bits).  bf16 parts sum to n32 exactly.  fp16 parts do when n32 >= 1/2; below
// that the last part may fall among fp16's subnormals, whose spacing is 2^-24,
// and the sum is then within 2^-25 of n32 (the distance bounds of the fp16
// passes add 2^-24 for it).  *ok = false when fp16 cannot hold the norm
// (n32 >= 2^15), *exact = false when the sum is not n32.
template <bool F16>
__device__ __forceinline__ void norm_parts(float n32, uint16_t *p, bool *ok, bool *exact) {
  p[0] = to16<F16>(n32);
  const float r1 = n32 - from16<F16>(p[0]);
  p[1] = to16<F16>(r1);
  const float r2 = r1 - from16<F16>(p[1]);
  p[2] = to16<F16>(r2);
  *ok = !F16 || n32 < 32768.f;
  *exact = !F16 || (*ok && r2 - from16<F16>(p[2]) == 0.f);
}

template <bool F16>
__global__ void __launch_bounds__(PW * 32)
    prep_rows_kernel(const float *__restrict__ x, long ld, int n, int d, float scale,
                     double *norm64, float *norm32, unsigned char *flags, float *resid,
                     uint16_t *packed, int Kp, uint16_t *normpart,
                     int normpart_mode, SetStats *stats, RowShift sh) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const long nwarps = (long)gridDim.x * PW;
  // per-warp running statistics, reduced once per block at the end
  float w_maxnorm = 0.f, w_maxres = 0.f;
  int w_exact = 1, w_nan = 0;
  const int cols = packed ? (Kp > d ? Kp : d) : d;
  const float inv = 1.f / scale;
  // vectorised path: 4 consecutive coordinates per lane (d % 4 == 0, aligned rows)
  const bool vec = (d % 4 == 0) && (ld % 4 == 0) && ((reinterpret_cast<uintptr_t>(x) & 15) == 0) &&
                   (!packed || Kp % 4 == 0);
  for (long row = (long)blockIdx.x * PW + wid; row < n; row += nwarps) {
    const float *xr = x + row * ld;
    const float *mr = row_mu(sh, row, d);
    // FP32 per element: exact for integer data (partial sums < 2^24), within
    // (d/32 + 6) ulp otherwise -- the certificate's error bound covers that
    float s = 0.f, r = 0.f;
    int exact = 1, bad = 0;
    if (vec) {
      for (int c = lane * 4; c < cols; c += 128) {
        float4 q4 = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c < d) q4 = __ldg(reinterpret_cast<const float4 *>(xr + c));
        if (mr && c < d) q4 = sub4(q4, __ldg(reinterpret_cast<const float4 *>(mr + c)));
        const float e[4] = {q4.x, q4.y, q4.z, q4.w};
        uint16_t hb[4];
#pragma unroll
        for (int t = 0; t < 4; t++) {
          const float v = e[t];
          hb[t] = to16<F16>(scale * v);
          if (c + t < d) {
            s = fmaf(v, v, s);
            exact &= (v == rintf(v)) && (fabsf(v) <= 256.f);
            bad |= !isfinite(v);
            const float dv = pack_err<F16>(v, inv, hb[t]);  // exact
            r = fmaf(dv, dv, r);
          }
        }
        if (packed && c < Kp) {
          uint2 w;
          w.x = (uint32_t)hb[0] | ((uint32_t)hb[1] << 16);
          w.y = (uint32_t)hb[2] | ((uint32_t)hb[3] << 16);
          *reinterpret_cast<uint2 *>(packed + row * Kp + c) = w;
        }
      }
    } else {
      for (int c = lane; c < cols; c += 32) {
        const float v = c < d ? (mr ? __fsub_rn(__ldg(xr + c), __ldg(mr + c)) : __ldg(xr + c))
                              : 0.f;
        const uint16_t h = to16<F16>(scale * v);
        if (c < d) {
          s = fmaf(v, v, s);
          exact &= (v == rintf(v)) && (fabsf(v) <= 256.f);
          bad |= !isfinite(v);
          const float dv = pack_err<F16>(v, inv, h);
          r = fmaf(dv, dv, r);
        }
        if (packed && c < Kp) packed[row * Kp + c] = h;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, o);
      r += __shfl_xor_sync(0xffffffffu, r, o);
      exact &= __shfl_xor_sync(0xffffffffu, exact, o);
      bad |= __shfl_xor_sync(0xffffffffu, bad, o);
    }
    exact &= (s <= kExactNorm2Max) && !bad;
    bool nok = true, nexact = true;
    if (normpart && lane < 16) {
      uint16_t val = to16<F16>(0.f);
      if (normpart_mode == 1) {
        uint16_t p[3];
        norm_parts<F16>((float)s, p, &nok, &nexact);
        val = lane < 3 ? p[lane] : val;
      } else if (normpart_mode == 2) {
        val = to16<F16>(lane < 3 ? 1.f : 0.f);
      }
      normpart[row * 16 + lane] = val;
    }
    const float rr = nok ? sqrtf(r) * (1.f + 1e-5f) : INFINITY;
    // exact class also needs every packed value and norm part to be exact,
    // which fp16 cannot promise for large values and norms
    if (F16) exact &= nok && nexact && r == 0.f;
    if (lane == 0) {
      if (norm64) norm64[row] = (double)s;
      if (norm32) norm32[row] = (float)s;
      if (flags) flags[row] = (unsigned char)exact;
      if (resid) resid[row] = rr;
    }
    if (!bad) {
      w_maxnorm = fmaxf(w_maxnorm, sqrtf(s) * (1.f + 1e-5f));
      w_maxres = fmaxf(w_maxres, rr);
    } else {
      w_nan++;
    }
    w_exact &= exact;
  }
  if (!stats) return;
  __shared__ float s_norm[PW], s_res[PW];
  __shared__ int s_exact[PW], s_nan[PW];
  if (lane == 0) {
    s_norm[wid] = w_maxnorm;
    s_res[wid] = w_maxres;
    s_exact[wid] = w_exact;
    s_nan[wid] = w_nan;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float mn = 0.f, mr = 0.f;
    int ex = 1, nn = 0;
    for (int w = 0; w < PW; w++) {
      mn = fmaxf(mn, s_norm[w]);
      mr = fmaxf(mr, s_res[w]);
      ex &= s_exact[w];
      nn += s_nan[w];
    }
    atomicMax(&stats->max_norm_bits, __float_as_uint(mn));
    atomicMax(&stats->max_resid_bits, __float_as_uint(mr));
    if (!ex) atomicAnd(&stats->all_exact, 0);
    if (nn) atomicAdd(&stats->n_nan, nn);
  }
}

// Eight lanes per row of at most 128 columns, four rows per warp step: each
// lane four consecutive coordinates per float4, all of a row's loads in flight
// before the conversions.  Same outputs as prep_rows_kernel.  HBM bound (4 d + 2
// Kp + 32 bytes a row) once the conversions are few: two values per
// conversion, the packing error from the packed word, and the tests for integers
// and for infinities only on rows that can be either (no packing error, a
// norm that is not finite).  1M + 10k rows, d = 128: 217 -> 150 us.
constexpr int LPR = 8, NIT = 128 / (4 * LPR);

struct RowOut {
  float s, rr;      // sum of squares, packing error of the row
  int exact, bad;   // exact class; an infinity or a NaN among the coordinates
};

// xr: the row (mr: its translation or null), prow / nrow: where its packed
// values and its norm block go (or null); rv = false: no row, nothing is
// written.  All 32 lanes of the warp call it, sl the lane's place in its row.
template <bool F16>
__device__ __forceinline__ RowOut prep_row8(const float *xr, const float *mr, bool rv, int d,
                                            int cols, float scale, float inv, uint16_t *prow,
                                            int Kp, uint16_t *nrow, int normpart_mode, int sl) {
  float4 q4s[NIT];
#pragma unroll
  for (int it = 0; it < NIT; it++) {
    const int c = sl * 4 + it * 4 * LPR;
    q4s[it] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (rv && c < d) q4s[it] = __ldg(reinterpret_cast<const float4 *>(xr + c));
    if (mr && c < d) q4s[it] = sub4(q4s[it], __ldg(reinterpret_cast<const float4 *>(mr + c)));
  }
  float s = 0.f, r = 0.f;
#pragma unroll
  for (int it = 0; it < NIT; it++) {
    const int c = sl * 4 + it * 4 * LPR;
    if (c >= cols) break;
    const float4 q4 = q4s[it];
    const float e[4] = {q4.x, q4.y, q4.z, q4.w};
    uint2 w;
    float h[4];
    if (F16) {
      const __half2 h0 = __floats2half2_rn(scale * e[0], scale * e[1]);
      const __half2 h1 = __floats2half2_rn(scale * e[2], scale * e[3]);
      const float2 f0 = __half22float2(h0), f1 = __half22float2(h1);
      h[0] = f0.x; h[1] = f0.y; h[2] = f1.x; h[3] = f1.y;
      w.x = *reinterpret_cast<const uint32_t *>(&h0);
      w.y = *reinterpret_cast<const uint32_t *>(&h1);
    } else {
      const __nv_bfloat162 h0 = __floats2bfloat162_rn(scale * e[0], scale * e[1]);
      const __nv_bfloat162 h1 = __floats2bfloat162_rn(scale * e[2], scale * e[3]);
      w.x = *reinterpret_cast<const uint32_t *>(&h0);
      w.y = *reinterpret_cast<const uint32_t *>(&h1);
      h[0] = __uint_as_float(w.x << 16); h[1] = __uint_as_float(w.x & 0xffff0000u);
      h[2] = __uint_as_float(w.y << 16); h[3] = __uint_as_float(w.y & 0xffff0000u);
    }
#pragma unroll
    for (int t = 0; t < 4; t++) {  // (columns past d are zeros and add nothing)
      s = fmaf(e[t], e[t], s);
      const float dv = fmaf(h[t], -inv, e[t]);  // exact
      r = fmaf(dv, dv, r);
    }
    if (rv && prow && c < Kp) *reinterpret_cast<uint2 *>(prow + c) = w;
  }
#pragma unroll
  for (int o = LPR / 2; o > 0; o >>= 1) {  // stays inside the row's lanes
    s += __shfl_xor_sync(0xffffffffu, s, o);
    r += __shfl_xor_sync(0xffffffffu, r, o);
  }
  RowOut out;
  out.s = s;
  out.bad = 0;
  out.exact = r == 0.f && s <= (float)kExactNorm2Max;  // an exact-class row packs exactly
  const bool fin = s <= 3.4e38f;  // (then every coordinate is finite)
  if (__any_sync(0xffffffffu, out.exact || !fin)) {
    int exact = 1, bad = 0;
#pragma unroll
    for (int it = 0; it < NIT; it++) {
      const float e[4] = {q4s[it].x, q4s[it].y, q4s[it].z, q4s[it].w};
#pragma unroll
      for (int t = 0; t < 4; t++) {
        exact &= (e[t] == rintf(e[t])) && (fabsf(e[t]) <= 256.f);
        bad |= !isfinite(e[t]);
      }
    }
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) {
      exact &= __shfl_xor_sync(0xffffffffu, exact, o);
      bad |= __shfl_xor_sync(0xffffffffu, bad, o);
    }
    out.exact &= exact;
    out.bad = bad;
  }
  bool nok = true, nexact = true;
  uint16_t part[3] = {0, 0, 0};
  if (normpart_mode == 1) {
    norm_parts<F16>(s, part, &nok, &nexact);
  } else if (normpart_mode == 2) {
    part[0] = part[1] = part[2] = to16<F16>(1.f);
  }
  out.rr = nok ? sqrtf(r) * (1.f + 1e-5f) : INFINITY;
  if (F16) out.exact &= nok && nexact;
  if (nrow && rv && sl < 2)  // the first two lanes: the row's 32 bytes
    reinterpret_cast<uint4 *>(nrow)[sl] =
        sl ? make_uint4(0, 0, 0, 0)
           : make_uint4((uint32_t)part[0] | (uint32_t)part[1] << 16, part[2], 0, 0);
  return out;
}

// a block's share of a set's statistics, added to it
struct SetAcc {
  float maxnorm = 0.f, maxres = 0.f;
  int exact = 1, nan = 0;
  __device__ __forceinline__ void row(const RowOut &o, int sl) {
    if (!o.bad) {
      maxnorm = fmaxf(maxnorm, sqrtf(o.s) * (1.f + 1e-5f));
      maxres = fmaxf(maxres, o.rr);
    } else if (sl == 0) {
      nan++;
    }
    exact &= o.exact;
  }
};

// (ends with a barrier: the scratch is free for the block's next set)
__device__ __forceinline__ void block_stats(SetAcc w, int wpb, SetStats *stats) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {  // the warp's rows
    w.maxnorm = fmaxf(w.maxnorm, __shfl_xor_sync(0xffffffffu, w.maxnorm, o));
    w.maxres = fmaxf(w.maxres, __shfl_xor_sync(0xffffffffu, w.maxres, o));
    w.exact &= __shfl_xor_sync(0xffffffffu, w.exact, o);
    w.nan += __shfl_xor_sync(0xffffffffu, w.nan, o);
  }
  __shared__ SetAcc part[PW];
  if (lane == 0) part[wid] = w;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < wpb; i++) {
      w.maxnorm = fmaxf(w.maxnorm, part[i].maxnorm);
      w.maxres = fmaxf(w.maxres, part[i].maxres);
      w.exact &= part[i].exact;
      w.nan += part[i].nan;
    }
    atomicMax(&stats->max_norm_bits, __float_as_uint(w.maxnorm));
    atomicMax(&stats->max_resid_bits, __float_as_uint(w.maxres));
    if (!w.exact) atomicAnd(&stats->all_exact, 0);
    if (w.nan) atomicAdd(&stats->n_nan, w.nan);
  }
  __syncthreads();
}

template <bool F16>
__global__ void __launch_bounds__(PW * 32)
    prep_rows_vec_kernel(const float *__restrict__ x, long ld, int n, int d, float scale,
                         double *norm64, float *norm32, unsigned char *flags, float *resid,
                         uint16_t *packed, int Kp, uint16_t *normpart,
                         int normpart_mode, SetStats *stats, RowShift sh) {
  constexpr int RPW = 32 / LPR;  // rows per warp step
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int sub = lane / LPR, sl = lane % LPR;
  const int wpb = (int)(blockDim.x >> 5);  // warps per block (<= PW)
  const long nwarps = (long)gridDim.x * wpb;
  const float inv = 1.f / scale;
  SetAcc acc;
  const int cols = packed ? (Kp > d ? Kp : d) : d;
  for (long rbase = ((long)blockIdx.x * wpb + wid) * RPW; rbase < n; rbase += nwarps * RPW) {
    const long row = rbase + sub;
    const bool rv = row < n;
    const RowOut o = prep_row8<F16>(
        x + row * ld, rv ? row_mu(sh, row, d) : nullptr, rv, d, cols, scale, inv,
        packed ? packed + row * Kp : nullptr, Kp, normpart ? normpart + row * 16 : nullptr,
        normpart_mode, sl);
    if (rv && sl == 0) {
      if (norm64) norm64[row] = (double)o.s;
      if (norm32) norm32[row] = o.s;
      if (flags) flags[row] = (unsigned char)o.exact;
      if (resid) resid[row] = o.rr;
    }
    if (rv) acc.row(o, sl);
  }
  if (stats) block_stats(acc, wpb, stats);
}

// The bases of many pairs in one launch (group.cu): 256-row chunks of the
// concatenated base, each inside one pair (a pair starts at a multiple of
// 256 rows).  A block takes consecutive chunks and adds its statistics
// to a pair's when it leaves it.  One launch per pair spent more of a short
// pair's time on the launch than on its rows: 64 pairs, 14.6M rows of d = 128: 3.8
// ms -> 1.72 (the HBM rate of a copy).
__global__ void __launch_bounds__(PW * 32)
    prep_group_base_kernel(const GroupPair *__restrict__ pairs, int np, int nchunk, int d, int Kp,
                           uint16_t *packed, uint16_t *normpart, SetStats *stats) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int sub = lane / LPR, sl = lane % LPR;
  const int c0 = (int)((long)blockIdx.x * nchunk / gridDim.x);
  const int c1 = (int)((long)(blockIdx.x + 1) * nchunk / gridDim.x);
  int p = 0, cur = -1;
  SetAcc acc;
  for (int c = c0; c < c1; c++) {
    const int r0 = c * 256;
    if (c == c0) {  // the pair of the first chunk (the last that starts at or before it)
      int hi = np - 1;
      while (p < hi) {
        const int mid = (p + hi + 1) >> 1;
        if (pairs[mid].boff <= r0) p = mid; else hi = mid - 1;
      }
    } else {
      while (p + 1 < np && pairs[p + 1].boff <= r0) p++;
    }
    if (p != cur) {
      if (cur >= 0) block_stats(acc, PW, stats + cur);
      acc = SetAcc();
      cur = p;
    }
    const int boff = pairs[p].boff, n = pairs[p].nb;
    const float *b = pairs[p].b;
    for (int i = wid * 4 + sub; i < 256; i += PW * 4) {
      const int loc = r0 - boff + i;
      const bool rv = loc < n;
      if (!__any_sync(0xffffffffu, rv)) break;
      const long row = r0 + i;
      const RowOut o = prep_row8<false>(b + (long)loc * d, nullptr, rv, d, Kp, 1.f, 1.f,
                                        packed + row * Kp, Kp,
                                        normpart ? normpart + row * 16 : nullptr,
                                        normpart ? 1 : 0, sl);
      if (rv) acc.row(o, sl);
    }
  }
  if (cur >= 0) block_stats(acc, PW, stats + cur);
}

// the queries of many pairs in one launch, and the pair of each
__global__ void __launch_bounds__(PW * 32)
    prep_group_queries_kernel(const GroupPair *__restrict__ pairs, int np, int nq, int d, int Kp,
                              float scale, double *norm64, unsigned char *flags, float *resid,
                              uint16_t *packed, uint16_t *normpart, int *qpair) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int sub = lane / LPR, sl = lane % LPR;
  const float inv = 1.f / scale;
  const long step = (long)gridDim.x * PW * 4;
  for (long rbase = ((long)blockIdx.x * PW + wid) * 4; rbase < nq; rbase += step) {
    const long row = rbase + sub;
    const bool rv = row < nq;
    int p = 0, hi = np - 1;  // the last pair that starts at or before the row
    while (p < hi) {
      const int mid = (p + hi + 1) >> 1;
      if (pairs[mid].qoff <= row) p = mid; else hi = mid - 1;
    }
    const RowOut o = prep_row8<false>(
        rv ? pairs[p].q + (row - pairs[p].qoff) * d : nullptr, nullptr, rv, d, Kp, scale, inv,
        packed + row * Kp, Kp, normpart ? normpart + row * 16 : nullptr, normpart ? 2 : 0, sl);
    if (rv && sl == 0) {
      norm64[row] = (double)o.s;
      flags[row] = (unsigned char)o.exact;
      resid[row] = o.rr;
      qpair[row] = p;
    }
  }
}

__global__ void __launch_bounds__(PW * 32)
    prep_split_kernel(const float *__restrict__ x, long ld, int n, int d, float scale, int layout,
                      double *norm64, float *norm32, unsigned char *flags, float *lonorm,
                      float *resid, __nv_bfloat16 *packed, int Kp1, __nv_bfloat16 *normpart,
                      int normpart_mode, SetStats *stats) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const long nwarps = (long)gridDim.x * PW;
  const int Kp = 3 * Kp1;
  float w_maxnorm = 0.f, w_maxres = 0.f, w_maxlo = 0.f;
  int w_exact = 1, w_nan = 0;
  for (long row = (long)blockIdx.x * PW + wid; row < n; row += nwarps) {
    const float *xr = x + row * ld;
    float s = 0.f, r = 0.f, l = 0.f;
    int exact = 1, bad = 0;
    for (int c = lane; c < Kp1; c += 32) {
      const float v = c < d ? __ldg(xr + c) : 0.f;
      const __nv_bfloat16 hi = __float2bfloat16_rn(v);
      const float rest = v - __bfloat162float(hi);             // exact
      const __nv_bfloat16 lo = __float2bfloat16_rn(rest);
      const float r2 = rest - __bfloat162float(lo);            // exact
      if (c < d) {
        s = fmaf(v, v, s);
        exact &= (v == rintf(v)) && (fabsf(v) <= 256.f);
        bad |= !isfinite(v);
        const float lf = __bfloat162float(lo);
        l = fmaf(lf, lf, l);
        r = fmaf(r2, r2, r);
      }
      const __nv_bfloat16 shi = __float2bfloat16_rn(scale * __bfloat162float(hi));
      const __nv_bfloat16 slo = __float2bfloat16_rn(scale * __bfloat162float(lo));
      __nv_bfloat16 *pr = packed + row * Kp;
      pr[c] = shi;
      pr[Kp1 + c] = layout == 0 ? shi : slo;
      pr[2 * Kp1 + c] = layout == 0 ? slo : shi;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, o);
      r += __shfl_xor_sync(0xffffffffu, r, o);
      l += __shfl_xor_sync(0xffffffffu, l, o);
      exact &= __shfl_xor_sync(0xffffffffu, exact, o);
      bad |= __shfl_xor_sync(0xffffffffu, bad, o);
    }
    exact &= (s <= kExactNorm2Max) && !bad;
    if (normpart && lane < 16) {
      __nv_bfloat16 val = __float2bfloat16_rn(0.f);
      if (normpart_mode == 1) {
        const float n32 = s;
        const __nv_bfloat16 hi = __float2bfloat16_rn(n32);
        const float r1 = n32 - __bfloat162float(hi);
        const __nv_bfloat16 mid = __float2bfloat16_rn(r1);
        const float r2 = r1 - __bfloat162float(mid);
        const __nv_bfloat16 lo = __float2bfloat16_rn(r2);
        val = lane == 0 ? hi : lane == 1 ? mid : lane == 2 ? lo : val;
      } else if (normpart_mode == 2) {
        val = __float2bfloat16_rn(lane < 3 ? 1.f : 0.f);
      }
      normpart[row * 16 + lane] = val;
    }
    const float rr = sqrtf(r) * (1.f + 1e-5f), ll = sqrtf(l) * (1.f + 1e-5f);
    if (lane == 0) {
      if (norm64) norm64[row] = (double)s;
      if (norm32) norm32[row] = s;
      if (flags) flags[row] = (unsigned char)exact;
      if (resid) resid[row] = rr;
      if (lonorm) lonorm[row] = ll;
    }
    if (!bad) {
      w_maxnorm = fmaxf(w_maxnorm, sqrtf(s) * (1.f + 1e-5f));
      w_maxres = fmaxf(w_maxres, rr);
      w_maxlo = fmaxf(w_maxlo, ll);
    } else {
      w_nan++;
    }
    w_exact &= exact;
  }
  if (!stats) return;
  __shared__ float s_norm[PW], s_res[PW], s_lo[PW];
  __shared__ int s_exact[PW], s_nan[PW];
  if (lane == 0) {
    s_norm[wid] = w_maxnorm;
    s_res[wid] = w_maxres;
    s_lo[wid] = w_maxlo;
    s_exact[wid] = w_exact;
    s_nan[wid] = w_nan;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float mn = 0.f, mr = 0.f, ml = 0.f;
    int ex = 1, nn = 0;
    for (int w = 0; w < PW; w++) {
      mn = fmaxf(mn, s_norm[w]);
      mr = fmaxf(mr, s_res[w]);
      ml = fmaxf(ml, s_lo[w]);
      ex &= s_exact[w];
      nn += s_nan[w];
    }
    atomicMax(&stats->max_norm_bits, __float_as_uint(mn));
    atomicMax(&stats->max_resid_bits, __float_as_uint(mr));
    atomicMax(&stats->max_lo_bits, __float_as_uint(ml));
    if (!ex) atomicAnd(&stats->all_exact, 0);
    if (nn) atomicAdd(&stats->n_nan, nn);
  }
}
}  // namespace

int prep_rows(const float *x, long ld, int n, int d, float scale, double *norm64,
              float *norm32, unsigned char *flags, float *resid,
              __nv_bfloat16 *packed_bf, int Kp, __nv_bfloat16 *normpart_bf,
              int normpart_mode, SetStats *stats, cudaStream_t st, int warps, int f16,
              RowShift shift) {
  uint16_t *packed = reinterpret_cast<uint16_t *>(packed_bf);
  uint16_t *normpart = reinterpret_cast<uint16_t *>(normpart_bf);
  if (n <= 0) return OK;
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    YG_CUDA(cudaGetDevice(&dev));
    YG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  }
  const long cap = (long)sms * 16;
  // eight lanes per row (four rows per warp step) when a row is at most 128
  // float4-aligned columns; one warp per row otherwise
  const int cols = packed ? (Kp > d ? Kp : d) : d;
  const bool vec = (d % 4 == 0) && (ld % 4 == 0) &&
                   ((reinterpret_cast<uintptr_t>(x) & 15) == 0) && (!packed || Kp % 4 == 0) &&
                   (!normpart || (reinterpret_cast<uintptr_t>(normpart) & 15) == 0) &&
                   (!shift.mu || (reinterpret_cast<uintptr_t>(shift.mu) & 15) == 0);
  if (shift.mu && !shift.row_inst && shift.rows_per_inst < 1) {
    set_error(E_ARG, "prep_rows: rows_per_inst = %d", shift.rows_per_inst);
    return E_ARG;
  }
  if (vec && cols <= 128) {
    const int wpb = warps >= 1 && warps <= PW ? warps : PW;
    long blocks = ceil_div(n, wpb * 4);
    if (blocks > cap * PW / wpb) blocks = cap * PW / wpb;
    auto kern = f16 ? prep_rows_vec_kernel<true> : prep_rows_vec_kernel<false>;
    kern<<<(unsigned)blocks, wpb * 32, 0, st>>>(x, ld, n, d, scale, norm64, norm32, flags, resid,
                                              packed, Kp, normpart, normpart_mode, stats, shift);
  } else {
    long blocks = ceil_div(n, PW);
    if (blocks > cap) blocks = cap;
    auto kern = f16 ? prep_rows_kernel<true> : prep_rows_kernel<false>;
    kern<<<(unsigned)blocks, PW * 32, 0, st>>>(x, ld, n, d, scale, norm64, norm32, flags, resid,
                                               packed, Kp, normpart, normpart_mode, stats, shift);
  }
  YG_LAUNCH_CHECK();
  return OK;
}

bool prep_group_ok(const GroupPair *hp, int np, int d, int Kp) {
  if (d % 4 != 0 || Kp > 128) return false;
  for (int i = 0; i < np; i++)
    if (((reinterpret_cast<uintptr_t>(hp[i].b) | reinterpret_cast<uintptr_t>(hp[i].q)) & 15) != 0 ||
        hp[i].boff % 256 != 0)
      return false;
  return true;
}

int prep_group(const GroupPair *pairs, int np, long brows, int nq, int d, int Kp, float qscale,
               __nv_bfloat16 *bpack, __nv_bfloat16 *bnorm, SetStats *stats, __nv_bfloat16 *qpack,
               __nv_bfloat16 *qnorm, double *qn64, unsigned char *qflag, float *qres, int *qpair,
               cudaStream_t st) {
  int dev = 0, sms = 0;
  YG_CUDA(cudaGetDevice(&dev));
  YG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int nchunk = (int)ceil_div(brows, 256);
  prep_group_base_kernel<<<(unsigned)imin(nchunk, sms * 16), PW * 32, 0, st>>>(
      pairs, np, nchunk, d, Kp, reinterpret_cast<uint16_t *>(bpack),
      reinterpret_cast<uint16_t *>(bnorm), stats);
  YG_LAUNCH_CHECK();
  prep_group_queries_kernel<<<(unsigned)std::min<long>(ceil_div(nq, PW * 4), (long)sms * 8),
                              PW * 32, 0, st>>>(
      pairs, np, nq, d, Kp, qscale, qn64, qflag, qres, reinterpret_cast<uint16_t *>(qpack),
      reinterpret_cast<uint16_t *>(qnorm), qpair);
  YG_LAUNCH_CHECK();
  return OK;
}

int prep_rows_split(const float *x, long ld, int n, int d, float scale, int layout,
                    double *norm64, float *norm32, unsigned char *flags, float *lonorm,
                    float *resid, __nv_bfloat16 *packed, int Kp1, __nv_bfloat16 *normpart,
                    int normpart_mode, SetStats *stats, cudaStream_t st) {
  if (n <= 0) return OK;
  int dev = 0, sms = 0;
  YG_CUDA(cudaGetDevice(&dev));
  YG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  long blocks = ceil_div(n, PW);
  if (blocks > (long)sms * 16) blocks = (long)sms * 16;
  prep_split_kernel<<<(unsigned)blocks, PW * 32, 0, st>>>(x, ld, n, d, scale, layout, norm64,
                                                          norm32, flags, lonorm, resid, packed,
                                                          Kp1, normpart, normpart_mode, stats);
  YG_LAUNCH_CHECK();
  return OK;
}

}  // namespace yg
