// Test shim: the small-k assignment's shape rule and shared-memory layout
// (km_tc_lay.h) for a CPU test.
#include "../yael_gb300/csrc/km_tc_lay.h"

using namespace yg::kmtc;

extern "C" int shim_tc_shape_ok(int d, int k) { return shape_ok(d, k); }

// out: total bytes, stages, sums, centroid rows, point rows, pairs
extern "C" void shim_tc_lay(int d, int k, int sums, long *out) {
  const Lay L = choose_lay(d, k, sums);
  out[0] = (long)L.total;
  out[1] = L.S;
  out[2] = L.fuse;
  out[3] = L.csm;
  out[4] = L.xs;
  out[5] = L.pairs;
}

// total bytes of a given form
extern "C" long shim_tc_total(int d, int k, int S, int fuse, int csm, int xs, int pairs) {
  return (long)make_lay((d + 63) / 64, (k + 31) / 32 * 32, S, fuse, k, d, csm, xs, pairs).total;
}
