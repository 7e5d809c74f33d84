// Shared-memory layout of the small-k assignment kernel (km_tc.cu), and the
// choice of its form for a shape.  Plain C++ (no CUDA), so the tests compile
// it on its own.
#pragma once
#include <stddef.h>

#ifdef __CUDACC__
#define YG_HD __host__ __device__
#else
#define YG_HD
#endif

namespace yg {

constexpr int kTcMaxK = 256;

namespace kmtc {

constexpr int NDEC = 16;              // decision warps
constexpr int A_BLK = 128 * 128;      // 128 rows x 64 16-bit columns
constexpr int A_SIDE = 128 * 32;      // 128 rows x 16 16-bit columns
constexpr size_t kSmemMax = 227 * 1024;
// band mask words per point (odd: no bank conflicts)
YG_HD constexpr int band_words(int N) { return (N >> 5) | 1; }

struct Lay {
  int nkb, N, S, fuse, csm, xs, pairs;
  size_t stage_bytes, x_off, ts_off, b_off, bside_off, cf_off, band_off, lst_off, pair_off, acc_off,
      cnt_off, bar_off, total;
};

// S: ring stages; fuse: the sums of an instance; csm: its FP32 centroid rows;
// xs: every stage also holds the tile's FP32 point rows (128 x d floats);
// pairs: (point, member) pairs listed per decision warp
YG_HD inline Lay make_lay(int nkb, int N, int S, int fuse, int k, int d, int csm, int xs,
                          int pairs) {
  Lay L;
  L.nkb = nkb; L.N = N; L.S = S; L.fuse = fuse; L.csm = csm; L.xs = xs; L.pairs = pairs;
  size_t off = 0;
  L.x_off = (size_t)nkb * A_BLK + A_SIDE;
  // the tile's per-point norm and packing error (128 x float2) after its rows
  L.ts_off = L.x_off + (xs ? (((size_t)128 * d * 4 + 1023) & ~(size_t)1023) : 0);
  L.stage_bytes = L.ts_off + 1024;
  off += (size_t)S * L.stage_bytes;
  L.b_off = off;     off += (size_t)nkb * N * 128;  // N % 32 == 0: 1024-aligned blocks
  L.bside_off = off; off += (size_t)N * 32;
  L.cf_off = off;    off += csm ? (size_t)N * d * 4 : 0;  // FP32 centroid rows (d % 4 == 0)
  L.band_off = off;  off += (size_t)2 * 128 * band_words(N) * 4;
  L.lst_off = off;   off += (size_t)256 * 4;  // the tile's moves: new and old centroids
  L.pair_off = off;  off += (size_t)NDEC * pairs * 8;  // pairs, then their distances
  off = (off + 15) & ~(size_t)15;
  L.acc_off = off;   off += fuse ? (size_t)k * d * 8 : 0;
  L.cnt_off = off;   off += fuse ? (size_t)k * 4 : 0;
  off = (off + 15) & ~(size_t)15;
  L.bar_off = off;   off += (size_t)(2 * S + 12) * 8 + 16;
  L.total = off + 1024;  // alignment slack of the 1024-byte aligned base
  return L;
}

// shapes the kernel takes: whole float4 rows of at most 192 coordinates with up
// to 256 centroids, of at most 256 with up to 128 (a ring of two stages beside
// the centroid tile)
inline bool shape_ok(int d, int k) {
  return d >= 4 && d % 4 == 0 && k >= 1 && k <= kTcMaxK && (d <= 192 || (d <= 256 && k <= 128));
}

// The form for a shape that shape_ok takes (sums: an instance's k x d sums are
// wanted in shared memory).  Staged rows and sums give way, point rows first, where a
// ring of two stages and a pair list of 32 would not fit beside them; then the
// longest list that leaves two stages, and the ring takes what is left, up to
// six.  A list is worth more than a third or fourth stage, staged rows more
// than the longer list (200k points, us an assignment, mixture of 4 k / of k / 4
// tight clusters): d = 128, k = 224, three stages and 64 pairs 137 / 303, four and 32
// 147 / 329; d = 84, k = 170, staged rows and 32 pairs 96 / 231, four stages
// and 64 pairs 124 / 241; but staged rows and no list (d = 80, k = 224) 89 / 227, three
// stages and 64 pairs 99 / 217.  d = 132 to 192 with k > 224 has room for 32.
inline Lay choose_lay(int d, int k, bool sums) {
  const int nkb = (d + 63) / 64, N = (k + 31) / 32 * 32;
  int fuse = sums, csm = (size_t)N * d * 4 <= 32 * 1024, xs = 1, S = 6, pairs = 64;
  auto fits = [&](int S_, int pairs_) {
    return make_lay(nkb, N, S_, fuse, k, d, csm, xs, pairs_).total <= kSmemMax;
  };
  if (!fits(2, 32)) xs = 0;
  if (!fits(2, 32)) csm = 0;
  if (!fits(2, 32)) fuse = 0;
  if (!fits(2, pairs)) pairs = 32;
  while (S > 2 && !fits(S, pairs)) S--;
  return make_lay(nkb, N, S, fuse, k, d, csm, xs, pairs);
}

}  // namespace kmtc
}  // namespace yg
