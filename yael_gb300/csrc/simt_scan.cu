// FP32 CUDA-core distance passes.
//   * rows_kernel: thresholds, running thresholds (k = 1) and the threshold
//     sample of the plain k-NN pipeline;
//   * simt_scan_kernel: lists of C entries per chunk, for many queries among few
//     rows (fp32_lists, knn.cu), for exact ties by the thousand, and for the
//     allocation-free call, whose scratch they bound.
// (See scan.cuh for the selection contract.)
#include <limits.h>
#include <math.h>

#include "scan.cuh"
#include "simt_tile.cuh"

namespace yg {

namespace {

// ---- rows_kernel ------------------------------------------------------------
// Bound by the FP32 pipe (62 TFLOP/s of three-register FFMA measured).  256 threads
// hold 16 TM query rows x 128 base rows, thread (tx, ty) rows ty + 16 i and columns
// tx + 16 j: a row belongs to one half-warp, so the selection needs no staging
// tile and no atomics.  Operand slices of 16 coordinates stay row-major in
// shared memory (pitch 20: 16 lanes reading 16 bytes each of consecutive rows
// use every bank twice) and arrive by cp.async three deep, which leaves the
// registers for two CTAs per SM: one computes while the other selects or waits.
// TM = 8: 1,000 x 100k, d = 100, thresholds: 0.70 ms for 128-row tiles staged in
// shared memory, one CTA per SM -> 0.52 (39 TFLOP/s); TM = 2 where 128-row tiles would
// leave SMs without one.
namespace rows {

constexpr int BN = 128, BK = 16, LD = BK + 4, NT = 256, NST = 3;

template <int TM>
constexpr size_t smem_floats() {
  return (size_t)NST * (16 * TM + BN) * LD + 4 * BN + 3 * 16 * TM;
}

__device__ __forceinline__ void cp16(float *dst, const float *src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(bytes));
}
__device__ __forceinline__ void cp4(float *dst, const float *src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(ok ? 4 : 0));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// One value per lane, ascending over the 16 lanes of each half-warp.
__device__ __forceinline__ float sort16(float x, int tx) {
#pragma unroll
  for (int k = 2; k <= 16; k <<= 1)
#pragma unroll
    for (int s = k >> 1; s > 0; s >>= 1) {
      const float y = __shfl_xor_sync(0xffffffffu, x, s);
      x = ((tx & s) == 0) == ((tx & k) == 0) ? fminf(x, y) : fmaxf(x, y);
    }
  return x;
}
// the 16 smallest of two ascending lists of 16, ascending
__device__ __forceinline__ float merge16(float a, float b, int tx) {
  float x = fminf(a, __shfl_xor_sync(0xffffffffu, b, 15));
#pragma unroll
  for (int s = 8; s > 0; s >>= 1) {
    const float y = __shfl_xor_sync(0xffffffffu, x, s);
    x = (tx & s) == 0 ? fminf(x, y) : fmaxf(x, y);
  }
  return x;
}

enum Mode : int { FIXED, RUNNING, SAMPLE };

template <int MODE, int TM, bool PAD>
__global__ void __launch_bounds__(NT, 2)
    rows_kernel(const float *__restrict__ Q, long ldq, int nq, const float *__restrict__ B,
                long ldb, int nb, int d, const float *__restrict__ bn, long bn_stride, int metric,
                int vq, int vb, ScanSel sel) {
  constexpr int BM = 16 * TM;
  extern __shared__ __align__(16) float smem[];
  float *Nrm = smem + NST * (BM + BN) * LD;  // [4][BN]: the norms of tile t in t & 3
  float *Thr = Nrm + 4 * BN;                 // [BM] thresholds (RUNNING: least value so far)
  float *Slk = Thr + BM;                     // [BM] RUNNING: slack
  int *Cnt = reinterpret_cast<int *>(Slk + BM);  // [BM] candidates
  const int tid = threadIdx.x, lane = tid & 31, tx = tid & 15, ty = tid >> 4;
  const unsigned hm = 0xffffu << (lane & 16), below = hm & ((1u << lane) - 1u);
  const long q0 = (long)blockIdx.x * BM;
  const int ntb = (int)ceil_div(nb, BN);
  const int t_begin = blockIdx.y * sel.tiles_per_chunk;
  const int t_end = imin(ntb, t_begin + sel.tiles_per_chunk);
  const int nk = (d + BK - 1) / BK, nit = (t_end - t_begin) * nk;

  for (int r = tid; r < BM; r += NT) {
    const bool ok = q0 + r < nq;  // (rows past the queries never hit)
    if (MODE == FIXED) Thr[r] = ok ? sel.thr[q0 + r] : NAN;
    if (MODE == RUNNING) {
      Thr[r] = ok ? INFINITY : -INFINITY;
      Slk[r] = ok ? sel.run_scale * run_slack(sel.run_eps[q0 + r]) : 0.f;
    }
    Cnt[r] = 0;
  }

  // Slices in flight: thread tid copies coordinates 4 (tid & 3) .. + 3 of rows
  // tid / 4 (+ 64) of the queries and of the base tile.
  const int lr = tid >> 2, lk = (tid & 3) * 4;
  const float *qsrc = Q + (q0 + lr) * ldq + lk, *bsrc = B + ((long)t_begin * BN + lr) * ldb + lk;
  int left = nb - (t_begin * BN + lr);  // base rows from this thread's on
  int st = t_begin, sk = 0, sb = 0;     // next slice to load: tile, slice, buffer
  auto stage = [&]() {
    if (st < t_end) {
      float *dst = smem + sb * (BM + BN) * LD + lr * LD + lk;
      const int k = sk * BK;
      const int kleft = imin(imax(d - k - lk, 0), 4);  // coordinates of this copy within d
      auto copy = [&](float *to, const float *from, const float *any, bool ok, int vec) {
        const int n = ok ? kleft : 0;
        if (vec) {
          cp16(to, n ? from : any, n * 4);
        } else {
#pragma unroll
          for (int z = 0; z < 4; z++) cp4(to + z, z < n ? from + z : any, z < n);
        }
      };
#pragma unroll
      for (int r = 0; r < BM; r += 64)
        if (BM >= 64 || lr < BM) copy(dst + r * LD, qsrc + r * ldq + k, Q, q0 + lr + r < nq, vq);
#pragma unroll
      for (int r = 0; r < BN; r += 64)
        copy(dst + (BM + r) * LD, bsrc + r * ldb + k, B, r < left, vb);
      if (sk == 0 && metric == METRIC_L2 && tid < BN) {
        const long j = (long)st * BN + tid;
        cp4(Nrm + (st & 3) * BN + tid, bn + (j < nb ? j * bn_stride : 0), j < nb);
      }
      if (++sk == nk) {
        sk = 0;
        st++;
        bsrc += BN * ldb;
        left -= BN;
      }
      if (++sb == NST) sb = 0;
    }
    cp_commit();
  };

  float acc[TM][8];
  float lst[TM];
#pragma unroll
  for (int i = 0; i < TM; i++) {
    lst[i] = INFINITY;
#pragma unroll
    for (int j = 0; j < 8; j++) acc[i][j] = 0.f;
  }
  stage();
  stage();
  int t = t_begin, kb = 0, buf = 0;
  for (int it = 0; it < nit; it++) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    stage();
    const float *As = smem + buf * (BM + BN) * LD + ty * LD;
    const float *Bs = smem + buf * (BM + BN) * LD + (BM + tx) * LD;
    if (++buf == NST) buf = 0;
    const int kleft = d - kb * BK;
#pragma unroll
    for (int kk = 0; kk < BK; kk += 4) {
      if (PAD && kk >= kleft) break;
      float4 a[TM];
#pragma unroll
      for (int i = 0; i < TM; i++)
        a[i] = *reinterpret_cast<const float4 *>(As + i * 16 * LD + kk);
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const float4 b = *reinterpret_cast<const float4 *>(Bs + j * 16 * LD + kk);
#pragma unroll
        for (int i = 0; i < TM; i++) {
          acc[i][j] = fmaf(a[i].x, b.x, acc[i][j]);
          acc[i][j] = fmaf(a[i].y, b.y, acc[i][j]);
          acc[i][j] = fmaf(a[i].z, b.z, acc[i][j]);
          acc[i][j] = fmaf(a[i].w, b.w, acc[i][j]);
        }
      }
    }
    if (++kb < nk) continue;
    kb = 0;

    // the tile's values v = ||b||^2 - 2 q.b (or q.b); columns past nb never hit
    const int j0 = t * BN;
    const float *nrm = Nrm + (t & 3) * BN;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int col = tx + 16 * j;
      const float bnj = metric == METRIC_L2 ? nrm[col] : 0.f;
#pragma unroll
      for (int i = 0; i < TM; i++) {
        if (metric == METRIC_L2) acc[i][j] = fmaf(-2.f, acc[i][j], bnj);
        if (j0 + col >= nb) acc[i][j] = NAN;
      }
    }
#pragma unroll
    for (int i = 0; i < TM; i++) {
      const int row = ty + 16 * i;
      float m = acc[i][0];
#pragma unroll
      for (int j = 1; j < 8; j++) m = fminf(m, acc[i][j]);
      if (MODE == SAMPLE) {
        if (sel.blockmin) {
          lst[i] = merge16(lst[i], sort16(fminf(m, INFINITY), tx), tx);
        } else {
#pragma unroll 1
          for (int j = 0; j < 8; j++) {
            const float lo = j & 1 ? (j & 2 ? acc[i][3] : acc[i][1]) : (j & 2 ? acc[i][2] : acc[i][0]);
            const float hi = j & 1 ? (j & 2 ? acc[i][7] : acc[i][5]) : (j & 2 ? acc[i][6] : acc[i][4]);
            lst[i] = merge16(lst[i], sort16(fminf(j & 4 ? hi : lo, INFINITY), tx), tx);
          }
        }
        continue;
      }
      int cnt = Cnt[row];
      float thr = Thr[row];
      __syncwarp();  // every lane has read the row's state before it changes
      if (MODE == RUNNING) {
        float mr = m;  // the row's least value in this tile (NaN: none)
#pragma unroll
        for (int s = 8; s > 0; s >>= 1) mr = fminf(mr, __shfl_xor_sync(0xffffffffu, mr, s));
        const float rmin = thr;
        thr = __fadd_ru(fminf(mr, rmin), Slk[row]);
        if (mr < rmin) {
          // every candidate so far above the new threshold: start over
          if (thr < rmin) cnt = 0;
          if (tx == 0) {
            Thr[row] = mr;
            Cnt[row] = cnt;
          }
        }
      }
      if (__any_sync(0xffffffffu, m <= thr)) {
        const long o = ((long)blockIdx.y * nq + q0 + row) * sel.cap;
#pragma unroll
        for (int j = 0; j < 8; j++) {  // increasing column over (j, tx)
          const bool hit = acc[i][j] <= thr;
          const unsigned b = __ballot_sync(0xffffffffu, hit) & hm;
          const int pos = cnt + __popc(b & below);
          if (hit && pos < sel.cap) {
            sel.candv[o + pos] = acc[i][j];
            sel.candi[o + pos] = j0 + tx + 16 * j + sel.id_off;
          }
          cnt += __popc(b);
        }
        if (tx == 0) Cnt[row] = cnt;
      }
    }
    __syncwarp();  // the rows' state is the half-warp's own
    t++;
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
      for (int j = 0; j < 8; j++) acc[i][j] = 0.f;
  }

#pragma unroll
  for (int i = 0; i < TM; i++) {
    const int row = ty + 16 * i;
    const long q = q0 + row;
    if (q >= nq) continue;
    const long o = (long)blockIdx.y * nq + q;
    if (MODE == SAMPLE) {
      sel.topv[o * 16 + tx] = lst[i];
    } else if (tx == 0) {
      // (no slack: the candidates tie, and the first has the least id.  Rows
      // that tie by the hundred, 20k x 5,000: 44.8 ms -> 0.8)
      sel.cnt[o] = MODE == RUNNING && Slk[row] == 0.f ? min(Cnt[row], 1) : Cnt[row];
      if (MODE == RUNNING && sel.run_thr) sel.run_thr[o] = __fadd_ru(Thr[row], Slk[row]);
    }
  }
}

template <int MODE, int TM, bool PAD>
int launch(const float *q, long ldq, int nq, const float *b, long ldb, int nb, int d,
           const float *bn, long bn_stride, int metric, const ScanSel &sel, cudaStream_t st) {
  const size_t smem = sizeof(float) * smem_floats<TM>();
  YG_CHECK(ensure_smem((const void *)rows_kernel<MODE, TM, PAD>, smem));
  const int vq = (ldq & 3) == 0 && ((uintptr_t)q & 15) == 0;
  const int vb = (ldb & 3) == 0 && ((uintptr_t)b & 15) == 0;
  const dim3 grid((unsigned)ceil_div(nq, 16 * TM), (unsigned)sel.nchunk);
  rows_kernel<MODE, TM, PAD><<<grid, NT, smem, st>>>(q, ldq, nq, b, ldb, nb, d, bn, bn_stride,
                                                     metric, vq, vb, sel);
  YG_LAUNCH_CHECK();
  return OK;
}

// PAD: a last slice of fewer than 16 coordinates, whose padding is not worked
// through (d = 100: 591 -> 517 us); a kernel of its own, as the test costs the
// others 2%.
template <int TM, bool PAD>
int dispatch(const float *q, long ldq, int nq, const float *b, long ldb, int nb, int d,
             const float *bn, long bn_stride, int metric, const ScanSel &sel, cudaStream_t st) {
  if (sel.mode == SCAN_TOPV)
    return launch<SAMPLE, TM, PAD>(q, ldq, nq, b, ldb, nb, d, bn, bn_stride, metric, sel, st);
  if (sel.run_eps)
    return launch<RUNNING, TM, PAD>(q, ldq, nq, b, ldb, nb, d, bn, bn_stride, metric, sel, st);
  return launch<FIXED, TM, PAD>(q, ldq, nq, b, ldb, nb, d, bn, bn_stride, metric, sel, st);
}

}  // namespace rows

// ---- simt_scan_kernel: 128 queries x 128 base rows per tile, 256 threads,
// 8x8 micro-tiles; the finished tile is staged in shared memory so that each
// query row is scanned by two threads in increasing base order
using namespace simt;

template <int C>
__global__ void __launch_bounds__(NT, 1)
    simt_scan_kernel(const float *__restrict__ Q, long ldq, int nq,
                     const float *__restrict__ B, long ldb, int nb, int d,
                     const float *__restrict__ bn, long bn_stride, int metric,
                     ScanSel sel) {
  extern __shared__ __align__(16) float smem[];
  float *St = smem + kOperandFloats;          // [BM][ST_LD]
  float *Lv = St + BM * ST_LD;                // [C][NT]
  int *Li = reinterpret_cast<int *>(Lv + C * NT);
  const int tid = threadIdx.x;
  const long q0 = (long)blockIdx.x * BM;
  const int ntb = (int)ceil_div(nb, BN);
  const int t_begin = blockIdx.y * sel.tiles_per_chunk;
  const int t_end = imin(ntb, t_begin + sel.tiles_per_chunk);

  // selection role: row sr, column half sh
  const int sr = tid & (BM - 1), sh = tid >> 7;
  const long qrow = q0 + sr;
  float lmax = INFINITY;
#pragma unroll
  for (int s = 0; s < C; s++) {
    Lv[s * NT + tid] = INFINITY;
    Li[s * NT + tid] = -1;
  }
  const int tx = tid & 15, ty = tid >> 4;

  for (int t = t_begin; t < t_end; ++t) {
    const long j0 = (long)t * BN;
    float acc[8][8];
    tile_mainloop(Q, ldq, nq, q0, B, ldb, nb, j0, d, smem, acc);

    // epilogue: v = ||b||^2 - 2 q.b (or q.b) into the staging tile
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int col = col_of(j, tx);
      const long jg = j0 + col;
      const bool ok = jg < nb;
      const float bnj = (ok && metric == METRIC_L2) ? __ldg(bn + jg * bn_stride) : 0.f;
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const int row = row_of(i, ty);
        const float v = metric == METRIC_L2 ? fmaf(-2.f, acc[i][j], bnj) : acc[i][j];
        St[row * ST_LD + col] = ok ? v : NAN;
      }
    }
    __syncthreads();

    // selection: row sr, columns [sh*64, sh*64+64), increasing base index
    if (qrow < nq) {
      const float *srow = St + sr * ST_LD + sh * 64;
      const int jbase = (int)(j0 + sh * 64);
      for (int c = 0; c < 64; c++) {
        const float v = srow[c];
        if (v < lmax) {
          int p = C - 1;
          while (p > 0 && Lv[(p - 1) * NT + tid] > v) {
            Lv[p * NT + tid] = Lv[(p - 1) * NT + tid];
            Li[p * NT + tid] = Li[(p - 1) * NT + tid];
            p--;
          }
          Lv[p * NT + tid] = v;
          Li[p * NT + tid] = jbase + c;
          lmax = Lv[(C - 1) * NT + tid];
        }
      }
    }
    __syncthreads();  // staging tile is rewritten by the next tile
  }

  if (sh == 0 && qrow < nq) {
    // merge the two half-row lists, lexicographic (v, id)
    int ia = 0, ib = 0;
    const long o = ((long)blockIdx.y * nq + qrow) * C;
    for (int s = 0; s < C; s++) {
      const float va = ia < C ? Lv[ia * NT + tid] : INFINITY;
      const float vb = ib < C ? Lv[ib * NT + tid + 128] : INFINITY;
      const int xa = ia < C ? Li[ia * NT + tid] : -1;
      const int xb = ib < C ? Li[ib * NT + tid + 128] : -1;
      const bool takeA =
          (ia < C) && (ib >= C || va < vb || (va == vb && (unsigned)xa <= (unsigned)xb));
      if (takeA) {
        sel.topv[o + s] = va;
        sel.topi[o + s] = xa < 0 ? xa : xa + sel.id_off;
        ia++;
      } else {
        sel.topv[o + s] = vb;
        sel.topi[o + s] = xb < 0 ? xb : xb + sel.id_off;
        ib++;
      }
    }
  }
}

template <int C>
int launch(const float *q, long ldq, int nq, const float *b, long ldb, int nb, int d,
           const float *bn, long bn_stride, int metric, const ScanSel &sel,
           cudaStream_t st) {
  const size_t smem = sizeof(float) * (kOperandFloats + BM * ST_LD) + (size_t)C * NT * 8;
  YG_CHECK(ensure_smem((const void *)simt_scan_kernel<C>, smem));
  dim3 grid((unsigned)ceil_div(nq, BM), (unsigned)sel.nchunk);
  simt_scan_kernel<C><<<grid, NT, smem, st>>>(q, ldq, nq, b, ldb, nb, d, bn,
                                                     bn_stride, metric, sel);
  YG_LAUNCH_CHECK();
  return OK;
}
}  // namespace

int simt_scan(const float *q, long ldq, int nq, const float *b, long ldb, int nb,
              int d, const float *bn, long bn_stride, int metric, const ScanSel &sel,
              cudaStream_t st) {
  if (nq <= 0 || nb <= 0) return OK;
  if (sel.mode != SCAN_TOPC) {
    const auto f = d % rows::BK ? (sel.tile_m == 32 ? rows::dispatch<2, true> : rows::dispatch<8, true>)
                                : (sel.tile_m == 32 ? rows::dispatch<2, false> : rows::dispatch<8, false>);
    return f(q, ldq, nq, b, ldb, nb, d, bn, bn_stride, metric, sel, st);
  }
  switch (sel.C) {
    case 2: return launch<2>(q, ldq, nq, b, ldb, nb, d, bn, bn_stride, metric, sel, st);
    case 4: return launch<4>(q, ldq, nq, b, ldb, nb, d, bn, bn_stride, metric, sel, st);
    case 8: return launch<8>(q, ldq, nq, b, ldb, nb, d, bn, bn_stride, metric, sel, st);
    case 16: return launch<16>(q, ldq, nq, b, ldb, nb, d, bn, bn_stride, metric, sel, st);
    case 32: return launch<32>(q, ldq, nq, b, ldb, nb, d, bn, bn_stride, metric, sel, st);
  }
  set_error(E_ARG, "simt_scan: unsupported list length C=%d", sel.C);
  return E_ARG;
}

// 128-row tiles where they give every SM one, else 32-row tiles
int simt_tile_m(int nq, int nb, int num_sms) {
  return ceil_div(nq, 128) * ceil_div(nb, SIMT_TILE_N) >= num_sms ? 128 : 32;
}

int choose_chunks(int n_query_tiles, int n_base_tiles, int num_sms, int ctas_per_sm,
                  int min_tiles_per_chunk) {
  const int slots = num_sms * ctas_per_sm;
  int maxc = n_base_tiles / imax(1, min_tiles_per_chunk);
  if (maxc < 1) maxc = 1;
  if (n_query_tiles >= 4 * slots) return 1;
  int best = 1;
  double best_eff = -1;
  for (int c = 1; c <= maxc && c <= 4096; c++) {
    const long total = (long)n_query_tiles * c;
    const long waves = (total + slots - 1) / slots;
    const double eff = (double)total / (double)(waves * slots);
    if (total >= slots && eff >= 0.9) return c;
    if (eff > best_eff + 1e-9) {
      best_eff = eff;
      best = c;
    }
    if (total >= 8L * slots) break;
  }
  return best;
}

}  // namespace yg
