// The fused "distance tile + per-query selection" pass.  Two producers of
// distance tiles share the selection contract:
//   * simt_scan  -- FP32 FFMA tiles on the CUDA cores (the plain path)
//   * tc_scan    -- BF16 tcgen05 tiles with FP32 accumulation in TMEM
// Both evaluate, for query row q and base row j,
//     v(q, j) = ||b_j||^2 - 2 q.b_j        (L2; ||q||^2 is added later)
//     v(q, j) = q.b_j                       (dot product)
// and never write the nq x nb matrix.  Selection modes:
//   TOPC   -- every (query, base chunk) keeps its C smallest (v, j) in
//             lexicographic order (strict '<' over increasing j), written to
//             topv/topi[(chunk * nq + q) * C + s], ascending.
//   THRESH -- every (q, j) with v <= thr[q] is appended to a candidate
//             region owned by one thread: region r = chunk * halves + column
//             half (halves = 2 for the tensor-core producer, whose two warps
//             of a row split the columns; 1 for the CUDA-core one), slots
//             candv/candi[(r * nq + q) * cap + s], count cnt[r * nq + q] (all
//             hits, including those that did not fit in cap).  No atomics:
//             each (region, query) has exactly one writer.
//             With run_eps (k = 1) the threshold is not given but runs:
//             the smallest v the region has seen plus run_slack(eps).  A
//             region starts over when its threshold falls below all its
//             candidates, so it ends with the few rows that can still be the
//             nearest; every row it left out is above its last threshold.
#pragma once
#include "common.cuh"

namespace yg {

struct SetStats;

// Grouped passes (tc_scan only): many (queries, base) pairs in one persistent
// launch.  The pairs' packed queries are concatenated, and so are their packed
// bases, each pair's base padded so that its tiles (in the view the pass
// reads) start at a tile boundary.  A unit is one query tile of one pair
// against a range of that pair's base tiles.
struct GroupUnit {
  int q0;              // first query row of the tile (concatenated rows)
  int qend;            // end of the pair's query rows
  int t_begin, t_end;  // base tiles of this view of the concatenated base
  int bend;            // end of the pair's valid columns in this view
  int pair;            // index into the pair table
  int chunk;           // chunk of the pair's base (THRESH region; 0 for lists)
  int blockmin;        // TOPV: the unit reads the sample in blocks (ScanSel::blockmin)
};

// Per pair: where its candidates go (THRESH) and what the re-rank needs.
struct GroupPair {
  long cnt_off;   // region counters: cnt[cnt_off + r * nq + (row - qoff)]
  long cand_off;  // slots: candv/candi[cand_off + (r * nq + (row - qoff)) * cap + s]
  int qoff, nq;   // the pair's rows in the concatenated queries
  int boff;       // first row of the pair in the concatenated base (ids are relative)
  int nb;
  int nreg;       // THRESH regions per query (chunks * halves)
  int cap;        // THRESH slots per region
  const float *q;           // the pair's query rows (FP32, stride d): exact re-rank
  const float *b;           // the pair's base rows (FP32, stride d)
  int *out_idx;             // the pair's outputs, nq x k
  float *out_dis;
  const SetStats *bs;       // the pair's base statistics
};

// SCAN_TOPV is SCAN_TOPC without ids (only the values are kept and written;
// used where a rank statistic of the distances is all that is needed).
enum ScanMode : int { SCAN_TOPC = 0, SCAN_THRESH = 1, SCAN_TOPV = 2 };
enum Metric : int { METRIC_L2 = 2, METRIC_DOT = 16 };

struct ScanSel {
  int mode = SCAN_TOPC;
  int C = 1;
  int nchunk = 1;           // base chunks
  int tiles_per_chunk = 1;  // base tiles per chunk
  float *topv = nullptr;
  int *topi = nullptr;
  const float *thr = nullptr;
  // THRESH: eps per query, thresholds run; they start from thr where it is given
  // (tc_scan)
  const float *run_eps = nullptr;
  // bounds of eps a running threshold leaves: twice as many in an FP32 pass,
  // whose eps is no larger than the FP32 re-rank's own error, which the
  // certificate takes off too (20k x 200, d = 128, unit rows: every iteration of
  // a k-means had rejected points, 3.60 ms for 8 iterations)
  float run_scale = 1.f;
  int *cnt = nullptr;
  float *candv = nullptr;
  int *candi = nullptr;
  int cap = 0;              // THRESH: slots per (region, query)
  int halves = 2;           // THRESH: regions per chunk (column halves of a row)
  int id_off = 0;           // added to every emitted base id (a pass over a base slice)
  // grouped pass (units != null): the work units, in launch order, and the
  // pair table; the pass's nq / nb are those of the concatenated operands
  const GroupUnit *units = nullptr;
  int nunits = 0;
  const GroupPair *gpairs = nullptr;
  int max_ctas = 0;         // persistent passes: grid limit (0 = one CTA per SM)
  // TOPV (tc_scan): the list holds minima of 32-row blocks of the sample
  // instead of single values; see kSampleSuper
  int blockmin = 0;
  // THRESH (tc_scan): well under one hit in 32 rows x 32 columns expected, or
  // nearly all of them hits: both are best drained a row of 32 at a time
  int queue = 0;
  // FP32 pass: query rows per tile (simt_tile_m); running thresholds: where a
  // region's last threshold goes ([region][query], may be null)
  int tile_m = 128;
  float *run_thr = nullptr;
  int f16 = 0;              // tensor-core passes: fp16 operands (else bf16)
  // tensor-core passes: bound of every wait (0: kWaitLimitNs), and a test
  // switch under which the producer issues no load, so that the consumers'
  // bounded waits expire (wait_limit_ns / test_withhold_loads in common.cuh)
  unsigned long long wait_ns = 0;
  int withhold = 0;
  __host__ __device__ int nregion() const { return nchunk * halves; }
};

// What a running threshold leaves above the smallest value: two error bounds
// (the row of the smallest exact distance is within them) and a little for the
// certificate's roundings.  Where no bound holds the rows nearest by value are
// kept all the same: they give the later passes a distance to start from.
__host__ __device__ inline float run_slack(float eps) {
  return eps < INFINITY ? 2.0005f * eps : 0.f;
}

// Block minima of a threshold sample.  The c-th smallest of the minima of
// disjoint blocks is an upper bound of the c-th smallest sampled value, and the
// minimum of 32 columns comes with the tensor-core pass's accumulator load, so
// the sample's lists take one insertion attempt per 32 values.  A block's rows
// are kSampleD sample rows apart inside super tiles of kSampleSuper rows, so
// that neighbours stored next to one another fall into different blocks; a
// sample is cut to whole super tiles and used this way from kSampleMin rows on
// (there the c <= 20 smallest values share a block rarely enough that the
// threshold's rank grows by less than a tenth).
constexpr int kSampleD = 32, kSampleSuper = 32 * kSampleD, kSampleMin = 4 * kSampleSuper;

// The rank of a sample of one row in stride = k / 3: 13, at which 1.6e-5 of the
// queries find fewer than k rows; 12 (1.7e-4, and a band pass for them) from a
// stride of 200 on, where the expected 13 strides come near the 8,192
// candidates that a query may have, and the queries past them go to the exhaustive
// pass: 200 queries, d = 64, 100k rows, k = 1,000: 4 of them at 13 (1.68 ms), none at 12
// (0.91); and where a rank of 13 leaves short bases without a sample: 20k rows,
// k = 1,200: 4.3 ms and 1.0.
inline int sample_rank_3(int stride) { return stride >= 200 ? 12 : 13; }

// FP32 CUDA-core producer.  q: nq rows (stride ldq floats); b: nb rows (stride
// ldb floats); bn: ||b||^2 as float with stride bn_stride (L2 only).
// Base tiles are 128 rows.  Reported base ids are j (row index in this view).
// THRESH regions are chunks (halves = 1); a TOPV pass with blockmin lists the
// minima of 8 rows.  TOPC: lists of 2 to 32 entries a chunk.
constexpr int SIMT_TILE_N = 128;
int simt_tile_m(int nq, int nb, int num_sms);
int simt_scan(const float *q, long ldq, int nq, const float *b, long ldb, int nb,
              int d, const float *bn, long bn_stride, int metric, const ScanSel &sel,
              cudaStream_t st);

// number of base chunks that gives enough CTAs for the GPU
int choose_chunks(int n_query_tiles, int n_base_tiles, int num_sms, int ctas_per_sm,
                  int min_tiles_per_chunk);

}  // namespace yg
