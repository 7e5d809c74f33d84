"""Exact k-NN parity on the GPU, through the C ABI.

The oracle is the FP64 brute force (canonical order: distance, then base id);
the reference's own outputs (tests/golden) are checked modulo its
heap-history tie order.  Every distance pass is covered: the plain FP32
CUDA-core path, the BF16 and FP16 tensor-core paths with exact re-rank and
the 3xBF16 split.
"""
import ctypes
import os

import numpy as np
import pytest

import yael_gb300 as yg
from _util import (GOLDEN, assign_mismatches, check_knn_ties, exact_dist64, knn_exact, knn_port,
                   ptr)
from yael_gb300 import synth

pytestmark = pytest.mark.gpu
PRECS = ["fp32", "bf16"]
NT = os.cpu_count() or 8


def gpu_knn(b, q, k, prec, dt=2):
    idx, dis, st = yg.knn(q, b, nnn=k, distance_type=dt, precision=prec, stats=True)
    return idx, dis, st


def assert_exact(b, q, k, prec, rtol=2e-6):
    idx, dis, st = gpu_knn(b, q, k, prec)
    ridx, rdis, r64 = knn_exact(b, q, k, NT)
    mism = np.nonzero((idx != ridx).any(1))[0]
    if len(mism):
        # only FP64-exact ties may differ (equal distance, different id order is impossible
        # with ties by id, so any mismatch is an error unless distances tie exactly)
        d_gpu = exact_dist64(b, q, idx)
        bad = check_knn_ties(idx, d_gpu, ridx, r64)
        assert bad == 0, f"{prec}: {len(mism)} rows differ, first {mism[:5]}"
    np.testing.assert_allclose(dis, rdis, rtol=rtol, atol=1e-6 * max(1.0, float(np.abs(rdis).max())))
    return st


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("k", [1, 5, 37])
def test_golden_integer_ties(prec, k):
    g = np.load(os.path.join(GOLDEN, "knn_int.npz"))
    b, q = g["b"], g["q"]
    idx, dis, st = gpu_knn(b, q, k, prec)
    ridx, rdis, r64 = knn_exact(b, q, k)
    np.testing.assert_array_equal(idx, ridx)          # canonical order, ties by id
    np.testing.assert_array_equal(dis, g[f"dis_k{k}"])  # exact integers, same as the reference
    assert check_knn_ties(g[f"idx_k{k}"], exact_dist64(b, q, g[f"idx_k{k}"]), idx, r64) == 0
    assert st["exact_class"] == 1


@pytest.mark.parametrize("prec", PRECS + ["fp16"])
def test_golden_float(prec):
    g = np.load(os.path.join(GOLDEN, "knn_float.npz"))
    assert_exact(g["b"], g["q"], 10, prec)
    idx, dis, _ = gpu_knn(g["b"], g["q"], 1, prec)
    np.testing.assert_array_equal(idx, g["idx_k1"])


@pytest.mark.parametrize("prec", ["bf16", "fp16"])
def test_k1_near_twin_rows(prec):
    """Base rows in pairs ~2e-7 of their norm apart (as an empty-cluster split
    leaves them): a query near a pair is a near tie in FP32, settled by the
    sign of the two distances' difference; ids identical to the FP64 oracle."""
    rng = np.random.default_rng(41)
    b0 = rng.standard_normal((6000, 64)).astype(np.float32)
    tw = rng.choice(6000, 1500, replace=False)
    e = (rng.standard_normal((1500, 64)) *
         (np.linalg.norm(b0[tw], axis=1, keepdims=True) * 1e-7)).astype(np.float32)
    b = np.concatenate([b0, b0[tw] - e]).astype(np.float32)
    b[tw] += e
    q = (b0[rng.choice(tw, 4000)] + 0.05 * rng.standard_normal((4000, 64))).astype(np.float32)
    idx, dis, _ = gpu_knn(b, q, 1, prec)
    ridx, rdis, _ = knn_exact(b, q, 1, NT)
    np.testing.assert_array_equal(idx, ridx)
    np.testing.assert_allclose(dis, rdis, rtol=5e-6, atol=1e-7)


@pytest.mark.parametrize("prec", PRECS + ["bf16x3", "fp16"])
@pytest.mark.parametrize("nq,nb,d,k", [(1, 1, 1, 1), (7, 5, 3, 5), (33, 300, 129, 17),
                                        (130, 2000, 64, 100), (300, 9000, 96, 33),
                                        (257, 1000, 7, 1), (64, 3000, 200, 250),
                                        (100, 5000, 300, 10)])
def test_shapes_gaussian(prec, nq, nb, d, k):
    rng = np.random.default_rng(nq * 7 + nb + d)
    b = rng.standard_normal((nb, d)).astype(np.float32)
    q = rng.standard_normal((nq, d)).astype(np.float32)
    assert_exact(b, q, k, prec)


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("k", [1, 10, 100])
def test_sift_like_medium(prec, k):
    b = synth.sift_like(120_000, 128, seed=1)
    q = synth.sift_like(300, 128, seed=2)
    idx, dis, st = gpu_knn(b, q, k, prec)
    ridx, rdis, _ = knn_exact(b, q, k, NT)
    np.testing.assert_array_equal(idx, ridx)
    np.testing.assert_array_equal(dis, rdis)
    assert st["exact_class"] == 1 and st["n_fallback"] == 0


@pytest.mark.parametrize("prec", PRECS + ["bf16x3", "fp16"])
def test_unit_vectors_oversampled(prec):
    b = synth.unit_gaussian(50_000, 128, seed=3)
    q = synth.unit_gaussian(200, 128, seed=4)
    st = assert_exact(b, q, 32, prec)
    assert st["n_fallback"] <= 2


@pytest.mark.parametrize("prec", PRECS)
def test_k_equals_nb_and_duplicates(prec):
    rng = np.random.default_rng(9)
    b = rng.integers(0, 3, (50, 4)).astype(np.float32)   # many exact duplicates
    q = rng.integers(0, 3, (20, 4)).astype(np.float32)
    for k in (50, 13, 1):
        idx, dis, _ = gpu_knn(b, q, k, prec)
        ridx, rdis, _ = knn_exact(b, q, k)
        np.testing.assert_array_equal(idx, ridx)
        np.testing.assert_array_equal(dis, rdis)


@pytest.mark.parametrize("k", [1, 10])
def test_fp16_rows_out_of_range_still_exact(k):
    """Rows fp16 cannot hold (here ||b||^2 up to ~6e6 > 2^15, and query values
    of 4e4 whose -2q overflows) get an infinite error bound: their queries
    fail the certificate and the later passes (3xBF16 band, FP64) settle them."""
    b = synth.sift_like(6000, 64, seed=21)
    q = synth.sift_like(50, 64, seed=22)
    q[::7, 3] = 4.0e4
    idx, dis, st = gpu_knn(b, q, k, "fp16")
    ridx, rdis, _ = knn_exact(b, q, k)
    np.testing.assert_array_equal(idx, ridx)
    np.testing.assert_array_equal(dis, rdis)
    assert st["n_band"] + st["n_second"] + st["n_fallback"] > 0


def test_nan_rows_follow_reference_padding():
    rng = np.random.default_rng(5)
    b = rng.standard_normal((400, 16)).astype(np.float32)
    q = rng.standard_normal((6, 16)).astype(np.float32)
    q[2, 3] = np.nan
    for k in (1, 4):
        idx, dis, _ = gpu_knn(b, q, k, "fp32")
        pidx, pdis = knn_port(b, q, k, nt=1)
        np.testing.assert_array_equal(idx[2], pidx[2])
        np.testing.assert_array_equal(dis[2].view(np.uint32), pdis[2].view(np.uint32))
        ok = [0, 1, 3, 4, 5]
        np.testing.assert_array_equal(idx[ok], knn_exact(b, q[ok], k)[0])


@pytest.mark.parametrize("prec", PRECS + ["fp16"])
@pytest.mark.parametrize("k", [7, 1])
def test_dot_product_metric(prec, k):
    """k = 1 takes the short re-rank's k = 1 form (reductions, FP32 certificate)."""
    rng = np.random.default_rng(6)
    b = rng.standard_normal((3000, 40)).astype(np.float32)
    q = rng.standard_normal((50, 40)).astype(np.float32)
    idx, dis, _ = gpu_knn(b, q, k, prec, dt=16)
    full = q.astype(np.float64) @ b.astype(np.float64).T
    order = np.lexsort((np.broadcast_to(np.arange(3000), full.shape), full), axis=1)[:, :k]
    np.testing.assert_array_equal(idx, order)
    np.testing.assert_allclose(dis, np.take_along_axis(full, order, 1), rtol=1e-5, atol=1e-5)


def test_weights_drop_in(gpu_lib):
    rng = np.random.default_rng(8)
    b = rng.standard_normal((800, 12)).astype(np.float32)
    q = rng.standard_normal((30, 12)).astype(np.float32)
    w = rng.uniform(0.5, 2.0, 800).astype(np.float32)
    idx = np.empty((30, 6), np.int32)
    dis = np.empty((30, 6), np.float32)
    gpu_lib.knn_full(2, 30, 800, 12, 6, ptr(b), ptr(q), ptr(w), ptr(idx), ptr(dis))
    full = ((q.astype(np.float64)[:, None] - b.astype(np.float64)[None]) ** 2).sum(-1) * w
    order = np.lexsort((np.broadcast_to(np.arange(800), full.shape), full), axis=1)[:, :6]
    np.testing.assert_array_equal(idx, order)


def test_drop_in_wrappers(gpu_lib):
    rng = np.random.default_rng(10)
    b = rng.standard_normal((500, 9)).astype(np.float32)
    v = rng.standard_normal((70, 9)).astype(np.float32)
    assign = np.empty(70, np.int32)
    s = gpu_lib.nn(70, 500, 9, ptr(b), ptr(v), ptr(assign))
    ridx, rdis, _ = knn_exact(b, v, 1)
    np.testing.assert_array_equal(assign, ridx[:, 0])
    assert abs(s - float(rdis.astype(np.float64).sum())) < 1e-4 * s
    idx = np.empty((70, 4), np.int32)
    p = gpu_lib.knn_thread(70, 500, 9, 4, ptr(b), ptr(v), ptr(idx), 8)
    dis = np.ctypeslib.as_array(ctypes.cast(p, ctypes.POINTER(ctypes.c_float)), shape=(70, 4)).copy()
    ctypes.CDLL(None).free(ctypes.c_void_p(p))
    np.testing.assert_array_equal(idx, knn_exact(b, v, 4)[0])
    np.testing.assert_allclose(dis, knn_exact(b, v, 4)[1], rtol=1e-5)


def test_cross_distances_vs_golden_and_fp64():
    g = np.load(os.path.join(GOLDEN, "cross.npz"))
    a, b = g["a"], g["b"]
    dis = yg.cross_distances(a, b)
    np.testing.assert_allclose(dis, g["dist2"], rtol=1e-5, atol=1e-4)
    full = ((b.astype(np.float64)[:, None] - a.astype(np.float64)[None]) ** 2).sum(-1)
    np.testing.assert_allclose(dis, full, rtol=1e-5, atol=1e-4)
    dot = yg.cross_distances(a, b, distance_type=16)
    np.testing.assert_allclose(dot, b.astype(np.float64) @ a.astype(np.float64).T, rtol=1e-5,
                               atol=1e-4)


def test_cross_distances_nonpacked_leaves_padding(gpu_lib):
    rng = np.random.default_rng(12)
    a = rng.standard_normal((20, 5)).astype(np.float32)
    b = rng.standard_normal((300, 5)).astype(np.float32)
    out = np.full((300, 25), 7.0, np.float32)  # ldd = 25 > na = 20
    gpu_lib.compute_cross_distances_nonpacked(5, 20, 300, ptr(a), 5, ptr(b), 5, ptr(out), 25)
    assert (out[:, 20:] == 7.0).all()
    full = ((b.astype(np.float64)[:, None] - a.astype(np.float64)[None]) ** 2).sum(-1)
    np.testing.assert_allclose(out[:, :20], full, rtol=1e-5, atol=1e-5)


def test_reorder_shortlist_and_recompute(gpu_lib):
    rng = np.random.default_rng(13)
    b = rng.standard_normal((1000, 24)).astype(np.float32)
    v = rng.standard_normal((40, 24)).astype(np.float32)
    idx = rng.integers(0, 1000, (40, 16)).astype(np.int32)
    idx[3, 10:] = -1  # short list stops at the first negative id
    dis = np.zeros((40, 16), np.float32)
    before = idx.copy()
    gpu_lib.knn_reorder_shortlist(40, 1000, 24, 16, ptr(b), ptr(v), ptr(idx), ptr(dis))
    for r in range(40):
        ki = 16 if r != 3 else 10
        d = ((v[r].astype(np.float64) - b[before[r, :ki]].astype(np.float64)) ** 2).sum(1)
        o = np.lexsort((np.arange(ki), d))
        np.testing.assert_array_equal(idx[r, :ki], before[r, :ki][o])
        np.testing.assert_allclose(dis[r, :ki], d[o], rtol=1e-6)
        np.testing.assert_array_equal(idx[r, ki:], before[r, ki:])
    # recompute over a base slice [label0, label0 + nb)
    srt = np.sort(rng.integers(0, 1000, (40, 8)), axis=1).astype(np.int32)
    kp = np.zeros(40, np.int32)
    d2 = np.zeros((40, 8), np.float32)
    gpu_lib.knn_recompute_exact_dists(40, 500, 24, 8, ptr(b), ptr(v), 0, ptr(kp), ptr(srt), ptr(d2))
    for r in range(40):
        n_in = int((srt[r] < 500).sum())
        assert kp[r] == n_in
        d = ((v[r].astype(np.float64) - b[srt[r, :n_in]].astype(np.float64)) ** 2).sum(1)
        np.testing.assert_array_equal(d2[r, :n_in], d.astype(np.float32))


def test_split_pass_settles_bf16_rejections():
    """Clustered float data with close neighbours: the BF16 certificate rejects
    many queries; the 3xBF16 second pass must settle them with exact ids."""
    v, _, _ = synth.gaussian_mixture(60000, 64, 30, 0.05, seed=31)
    q, _, _ = synth.gaussian_mixture(400, 64, 30, 0.05, seed=31)
    st = assert_exact(v, q, 1, "bf16")
    assert st["n_fallback"] <= 5
    st = assert_exact(v, q, 3, "bf16")
    assert st["n_fallback"] <= 5


def shell_data(nb=4000, nq=64, d=64, seed=41):
    """Base rows on thin shells around a far-away centre: the BF16 error bound
    dwarfs the spread of the distances, so every later-chance pass runs."""
    rng = np.random.default_rng(seed)
    c = rng.standard_normal(d) * 3.0
    u = rng.standard_normal((nb, d))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    r = 1.0 + 0.5 * rng.random(nb)
    b = (c + r[:, None] * u).astype(np.float32)
    q = (c + 1e-3 * rng.standard_normal((nq, d))).astype(np.float32)
    return b, q


@pytest.mark.parametrize("prec", ["fp32", "bf16", "bf16x3", "fp16"])
@pytest.mark.parametrize("k", [1, 5])
def test_later_chance_chain(prec, k):
    b, q = shell_data()
    st = assert_exact(b, q, k, prec)
    assert st["n_fallback"] <= 2
    if prec == "bf16":
        assert st["n_band"] > 0 and st["n_second"] > 0


def test_cta_pair_kernel_matches():
    """The CTA-pair form of the tensor-core pass (tcgen05 cta_group::2, chosen
    with YAEL_GPU_TC_PAIR=1) gives the same exact results; run in a child
    process since the switch is read once per process."""
    import subprocess
    import sys
    code = (
        "import numpy as np, sys; sys.path.insert(0, 'tests');"
        "from _util import knn_exact; import yael_gb300 as yg;"
        "rng = np.random.default_rng(77);"
        "b = rng.standard_normal((20000, 128)).astype(np.float32);"
        "q = rng.standard_normal((700, 128)).astype(np.float32);"
        "i1, d1 = yg.knn(q, b, nnn=10, precision='bf16');"
        "i2, d2 = yg.knn(q, b, nnn=1, precision='bf16x3');"
        "r1 = knn_exact(b, q, 10)[0]; r2 = knn_exact(b, q, 1)[0];"
        "assert (i1 == r1).all() and (i2 == r2).all(); print('pair ok')")
    env = dict(os.environ, YAEL_GPU_TC_PAIR="1")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, env=env, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and "pair ok" in r.stdout, r.stdout + r.stderr


@pytest.mark.parametrize("k", [1, 8, 100])
def test_host_upload_in_parts(k):
    """Host arrays with a large base go up in parts overlapped with the passes
    (thresholds from the first part); ids are still exact, including a base
    whose parts differ (sorted rows: part 0 is not representative)."""
    rng = np.random.default_rng(91)
    nb, nq, d = 300_000, 300, 64
    b = rng.standard_normal((nb, d)).astype(np.float32)
    b = b[np.argsort(b[:, 0])]  # ordered rows: a worst case for the first-part sample
    q = rng.standard_normal((nq, d)).astype(np.float32)
    idx, dis, st = gpu_knn(b, q, k, "bf16")
    ridx, rdis, r64 = knn_exact(b, q, k, NT)
    mism = np.nonzero((idx != ridx).any(1))[0]
    if len(mism):
        assert check_knn_ties(idx, exact_dist64(b, q, idx), ridx, r64) == 0
    np.testing.assert_allclose(dis, rdis, rtol=2e-6, atol=1e-5)


@pytest.mark.parametrize("nq,nb,d", [(1, 300, 16), (130, 20_000, 128), (20_000, 5000, 33)])
def test_fp32_nearest_first_pass(nq, nb, d):
    """k = 1 in FP32, settled by the first pass: rows whose exact distances tie
    by the hundred (more than a region holds), and unit rows, whose distances
    and dot products carry a rounding as large as the pass's."""
    rng = np.random.default_rng(nb)
    c = rng.integers(0, 9, (17, d)).astype(np.float32)
    b, q = c[rng.integers(0, 17, nb)], c[rng.integers(0, 17, nq)]
    st = assert_exact(b, q, 1, "fp32")
    assert st["exact_class"] == 1 and st["n_band"] == 0 and st["n_fallback"] == 0
    b = rng.standard_normal((nb, d)).astype(np.float32)
    q = rng.standard_normal((nq, d)).astype(np.float32)
    b /= np.linalg.norm(b, axis=1, keepdims=True)
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    assert assert_exact(b, q, 1, "fp32")["n_band"] == 0
    idx, _, st = gpu_knn(b, q, 1, "fp32", dt=16)
    dots = q.astype(np.float64) @ b.astype(np.float64).T
    np.testing.assert_array_equal(idx[:, 0], np.argmin(dots, axis=1))
    assert st["n_band"] == 0 and st["n_fallback"] == 0


@pytest.mark.parametrize("prec", ["bf16", "fp16", "bf16x3"])
@pytest.mark.parametrize("nq,nb", [(19_500, 200), (20_001, 287), (40_000, 1031), (77_900, 2049),
                                   (20_000, 4099), (80_000, 3900)])
def test_nearest_running_thresholds(nq, nb, prec):
    """k = 1 over enough queries for the running thresholds, at the edges of
    tiles, chunks and regions: rows in ascending and in descending distance, many
    equal rows (more than a region holds), NaN and infinite queries."""
    d = 20
    rng = np.random.default_rng(nb)
    b = rng.standard_normal((nb, d)).astype(np.float32)
    q = (b[rng.integers(0, nb, nq)] + 0.3 * rng.standard_normal((nq, d))).astype(np.float32)
    m = nq // 8
    b[nb // 2:nb // 2 + 40] = b[nb // 2]              # equal rows, near all of these queries
    q[:m] = b[nb // 2] + 0.01 * q[:m]
    b[40:120] = np.linspace(4, 0.1, 80, dtype=np.float32)[:, None]   # ever nearer, then farther
    b[120:200] = np.linspace(0.1, 4, 80, dtype=np.float32)[:, None]
    q[m:2 * m] = 1e-3 * q[m:2 * m]
    idx, dis, _ = gpu_knn(b, q, 1, prec)
    assert assign_mismatches(q, b, idx[:, 0].copy(), NT)[0] == 0
    np.testing.assert_allclose(dis[:, 0], ((q - b[idx[:, 0]]) ** 2).sum(1), rtol=2e-5, atol=1e-6)
    # integers: exact values, the lowest id of each group of equal rows
    bi = rng.integers(0, 3, (nb, d)).astype(np.float32)
    bi[nb - 60:] = bi[:60]
    qi = rng.integers(0, 3, (nq, d)).astype(np.float32)
    qi[:m] = bi[nb - 1]
    idx, _, st = gpu_knn(bi, qi, 1, prec)
    assert st["exact_class"] == 1
    assert assign_mismatches(qi, bi, idx[:, 0].copy(), NT)[0] == 0
    # queries without a nearest row
    q[5], q[nq - 1, 3] = np.nan, np.inf
    idx2, dis2, _ = gpu_knn(b, q, 1, prec)
    sel = np.setdiff1d(np.arange(nq), [5, nq - 1])
    ref1, _, _ = gpu_knn(b, q[[5, nq - 1]], 1, prec)
    np.testing.assert_array_equal(idx2[[5, nq - 1]], ref1)
    assert assign_mismatches(q[sel], b, idx2[sel, 0].copy(), NT)[0] == 0


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("nq,nb,k", [(300, 420, 20), (257, 8192, 100), (513, 1716, 100),
                                     (130, 3000, 20), (129, 8193, 50)])
def test_short_base_thresholds(nq, nb, k, prec):
    """More than sixteen neighbours in bases of a few thousand rows: thresholds
    from the shortest samples, clustered and sorted rows (samples that mislead)."""
    rng = np.random.default_rng(nb + k)
    b = rng.standard_normal((nb, 24)).astype(np.float32)
    q = rng.standard_normal((nq, 24)).astype(np.float32)
    assert_exact(b, q, k, prec)
    b[::max(1, k // 3)] *= 3                      # the sampled rows are the far ones
    assert_exact(b, q, k, prec)
    b = b[np.argsort((b ** 2).sum(1), kind="stable")].copy()
    assert_exact(b, q, k, prec)


@pytest.mark.parametrize("nq,nb,d,k", [(1, 130, 7, 1), (33, 1, 5, 1), (31, 600, 16, 2),
                                       (129, 127, 33, 1), (700, 9000, 17, 1), (64, 5000, 100, 5),
                                       (2000, 40_000, 12, 10), (300, 2200, 65, 3)])
def test_fp32_row_tiles(nq, nb, d, k):
    """The FP32 pass at the edges of its tiles, slices and chunks: aligned and
    unaligned rows, running thresholds in one and in many regions, samples in
    single values and in minima; clustered, integer and repeated rows."""
    rng = np.random.default_rng(nq + nb)
    b = rng.standard_normal((nb, d)).astype(np.float32)
    q = rng.standard_normal((nq, d)).astype(np.float32)
    assert_exact(b, q, k, "fp32")
    bi, qi = np.round(b).astype(np.float32), np.round(q).astype(np.float32)
    bi[nb // 2:] = bi[:nb - nb // 2]
    st = assert_exact(bi, qi, k, "fp32")
    assert st["exact_class"] == 1
    b = b[np.argsort(-(b ** 2).sum(1), kind="stable")].copy()
    assert_exact(b, q, k, "fp32")
    idx, _, _ = gpu_knn(b, q, k, "fp32", dt=16)
    dots = q.astype(np.float64) @ b.astype(np.float64).T
    np.testing.assert_array_equal(idx, np.argsort(dots, axis=1, kind="stable")[:, :k])


def fp64_order(q, b, k, dt=2):
    """The k smallest (FP64 distance, id), NaN never selected: ids, -1 past the
    rows that have a distance; k = 1: none that FP32 does not hold (yael/nn.c:404-407)."""
    q64, b64 = q.astype(np.float64), b.astype(np.float64)
    with np.errstate(all="ignore"):
        full = q64 @ b64.T if dt == 16 else ((q64[:, None] - b64[None]) ** 2).sum(2)
    key = np.where(np.isnan(full), np.inf, full)
    ids = np.broadcast_to(np.arange(len(b)), full.shape)
    order = np.lexsort((ids, key, np.isnan(full)), axis=1)[:, :k]
    got = np.take_along_axis(full, order, 1)
    bad = ~(got < 3.4e38) if k == 1 else np.isnan(got)
    return np.where(bad, -1, order)


@pytest.mark.parametrize("prec", ["fp16", "bf16x3"])
@pytest.mark.parametrize("nb,k", [(24, 20), (6, 1), (3000, 8), (3000, 30)])
def test_dot_product_infinite_rows(nb, k, prec):
    """Inner products with infinite rows: -inf where the 16-bit operands give NaN
    (a query value that is zero in fp16, the low part of an infinity)."""
    rng = np.random.default_rng(nb + k)
    b = rng.standard_normal((nb, 8)).astype(np.float32)
    q = (1 + rng.random((40, 8))).astype(np.float32)
    q[:, 5] = 1e-9
    b[nb // 2, 5], b[nb // 3, 2], b[nb - 1, 5] = -np.inf, np.inf, -np.inf
    idx, _, _ = gpu_knn(b, q, k, prec, dt=16)
    np.testing.assert_array_equal(idx, fp64_order(q, b, k, 16))


@pytest.mark.parametrize("dt", [2, 16])
@pytest.mark.parametrize("prec", ["fp32", "bf16", "fp16", "bf16x3"])
@pytest.mark.parametrize("nb,inf,k", [(10, 2, 9), (10, 2, 10), (24, 6, 20), (24, 0, 20), (10, 0, 9),
                                      (1, 1, 1), (6, 5, 1), (600, 595, 8), (300, 290, 20)])
def test_short_bases_infinite_rows(nb, inf, k, prec, dt):
    """Bases in which every row is a candidate, with rows that have infinite
    coordinates of either sign: (distance, id) order up to and past the
    finite rows; a finite base needs no later pass."""
    rng = np.random.default_rng(nb + k)
    b = rng.standard_normal((nb, 8)).astype(np.float32)
    q = (1 + rng.random((40, 8))).astype(np.float32)
    rows = np.sort(rng.permutation(nb)[:inf])
    b[rows, rng.integers(0, 8, inf)] = np.where(np.arange(inf) % 2, -np.inf, np.inf)
    q[:, 5] = 1e-9                # nothing in fp16, where it meets an infinity as 0 x inf
    idx, _, st = gpu_knn(b, q, k, prec, dt=dt)
    np.testing.assert_array_equal(idx, fp64_order(q, b, k, dt))
    if inf == 0:
        assert st["n_band"] == 0 and st["n_fallback"] == 0


@pytest.mark.parametrize("prec", ["fp32", "bf16", "fp16", "bf16x3"])
@pytest.mark.parametrize("nb,near,k", [(7, 0, 1), (7, 0, 5), (24, 0, 20), (600, 3, 8), (200, 7, 20)])
def test_short_bases_overflowing_distances(nb, near, k, prec):
    """Finite rows and queries whose norms are finite in FP32 and whose squared
    distances are not (1.6e19 against 0.6e19 the other way): ids in FP64 order,
    also where the list of a chunk is full of overflowed values."""
    rng = np.random.default_rng(nb)
    u = rng.standard_normal(8)
    u /= np.linalg.norm(u)
    q = (1.6e19 * u * (1 + 1e-2 * rng.random((20, 1)))).astype(np.float32)
    b = (-0.6e19 * u * rng.uniform(0.9, 1.1, (nb, 1))).astype(np.float32)
    b[rng.permutation(nb)[:near]] *= -1
    idx, _, _ = gpu_knn(b, q, k, prec)
    np.testing.assert_array_equal(idx, fp64_order(q, b, k))


@pytest.mark.parametrize("prec", ["fp32", "bf16", "fp16"])
@pytest.mark.parametrize("k", [1, 5])
@pytest.mark.parametrize("nq,nb,copies", [(1, 5000, 20), (3, 100_000, 17), (3, 100_000, 300),
                                          (40, 30_000, 100), (200, 9000, 300)])
def test_copies_of_a_row_need_no_exhaustive_pass(nq, nb, copies, k, prec):
    """Real-valued rows, one of them repeated side by side more often than a
    candidate region holds, next to every query: settled by the band passes."""
    rng = np.random.default_rng(nb + copies)
    b = rng.standard_normal((nb, 24)).astype(np.float32)
    r = nb // 3
    b[r:r + copies] = b[r]
    q = (b[r] + 0.05 * rng.standard_normal((nq, 24))).astype(np.float32)
    st = assert_exact(b, q, k, prec)
    assert st["n_fallback"] == 0


@pytest.mark.parametrize("prec", ["fp32", "bf16", "fp16"])
@pytest.mark.parametrize("nq,nb,d,k", [(300, 200_000, 32, 200), (1500, 60_000, 64, 10)])
@pytest.mark.parametrize("order", [1, -1])
def test_bases_in_norm_order(nq, nb, d, k, order, prec):
    """Inner products over a base stored in the order of its norms: the nearest
    rows lie together, and the first pass settles nearly every query."""
    rng = np.random.default_rng(nb)
    b = rng.standard_normal((nb, d)).astype(np.float32)
    b /= np.linalg.norm(b, axis=1, keepdims=True)
    b *= np.linspace(0.02, 4, nb, dtype=np.float32)[::order, None]
    q = rng.standard_normal((nq, d)).astype(np.float32)
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    idx, _, st = gpu_knn(b, q, k, prec, dt=16)
    dots = q.astype(np.float64) @ b.astype(np.float64).T
    near = np.sort(np.argpartition(dots, k, axis=1)[:, :k], axis=1)
    order = np.argsort(np.take_along_axis(dots, near, 1), axis=1, kind="stable")
    np.testing.assert_array_equal(idx, np.take_along_axis(near, order, 1))
    # (a query whose sample has fewer than its share of the near rows may need a
    # band pass: 2e-5 of them)
    assert st["n_band"] <= 2 and st["n_second"] == 0 and st["n_fallback"] == 0


@pytest.mark.parametrize("k", [2, 5, 10, 16, 17])
@pytest.mark.parametrize("nq,nb", [(1, 60_000), (300, 60_000), (2000, 9000)])
def test_fp32_copies_of_integer_rows(nq, nb, k):
    """A base of copies of 17 integer rows: thousands of rows tie with the k-th,
    and the least ids are the answer.  Up to 16 neighbours need no exhaustive
    pass in FP32."""
    rng = np.random.default_rng(nb)
    c = rng.integers(0, 9, (17, 20)).astype(np.float32)
    b, q = c[rng.integers(0, 17, nb)], c[rng.integers(0, 17, nq)]
    st = assert_exact(b, q, k, "fp32")
    assert st["exact_class"] == 1
    assert k > 16 or st["n_fallback"] == 0
    # queries that are not integers: no value is exact
    assert_exact(b, (q[:8] + 0.25).astype(np.float32), k, "fp32")


def test_tile_heights_are_tuned_apart():
    """FP32 passes over 32-row and over 128-row query tiles with the same number of
    tiles (256 and 1,024 queries: eight) choose their chunk counts by themselves (child
    process: the trace is switched on by the environment)."""
    import subprocess
    import sys
    code = (
        "import numpy as np, yael_gb300 as yg;"
        "rng = np.random.default_rng(7);"
        "b = rng.standard_normal((5120, 16)).astype(np.float32);"
        "q = rng.standard_normal((1024, 16)).astype(np.float32);"
        "[yg.knn(q[:n], b, nnn=1, precision='fp32') for n in (256, 1024) for _ in range(6)]")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True,
                       env=dict(os.environ, YAEL_GPU_TRACE="1"), timeout=300)
    assert r.returncode == 0, r.stderr
    assert r.stderr.count("autotune kind=4 key=(8,40,") == 2, r.stderr[-2000:]


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("nq,nb", [(300, 5000), (20_000, 5000), (40, 30_000), (7, 257)])
def test_nearest_among_copies_of_integer_rows(nq, nb, prec):
    """k = 1, exact values, hundreds of rows that tie with the nearest: the least
    id, from short and from long candidate lists and from thresholds."""
    rng = np.random.default_rng(nq)
    c = rng.integers(0, 9, (17, 33)).astype(np.float32)
    b, q = c[rng.integers(0, 17, nb)], c[rng.integers(0, 17, nq)]
    st = assert_exact(b, q, 1, prec)
    assert st["exact_class"] == 1 and st["n_band"] == 0 and st["n_fallback"] == 0


@pytest.mark.parametrize("d", [900, 3000, 6002])
@pytest.mark.parametrize("dt", [2, 16])
def test_near_ties_in_long_rows(d, dt):
    """Rows whose distances differ by 1e-12 to 1e-7 of their value, long enough that
    the roundings of pairs of floats add up: ids in FP64 order."""
    rng = np.random.default_rng(d)
    q = rng.standard_normal((6, d)).astype(np.float32)
    base = rng.standard_normal(d).astype(np.float32)
    b = np.repeat(base[None], 400, 0)
    b[:, 0] += np.linspace(-1e-6, 1e-6, 400).astype(np.float32)
    b[rng.permutation(400)[:200], d - 1] += np.float32(1e-6)
    idx, _, _ = gpu_knn(b, q, 30, "fp32", dt=dt)
    q64, b64 = q.astype(np.float64), b.astype(np.float64)
    full = q64 @ b64.T if dt == 16 else np.array([((x - b64) ** 2).sum(1) for x in q64])
    got = np.take_along_axis(full, idx, 1)
    # (the k smallest in FP64, in an order that FP64 sums in any order agree with)
    slack = 1e-13 * np.abs(full).max()
    assert (got <= np.sort(full, 1)[:, 29:30] + slack).all()
    assert (np.diff(got, axis=1) >= -slack).all()


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("nb,k", [(100_000, 1000), (20_000, 1200), (20_000, 610)])
def test_long_neighbour_lists_stay_within_the_candidates(nb, k, prec):
    """A thousand neighbours and more: the expected candidates come near the limit of
    a query's, and queries past it end in the exhaustive pass.  A few may, by the
    sample's luck."""
    rng = np.random.default_rng(nb)
    b = rng.standard_normal((nb, 64)).astype(np.float32)
    q = rng.standard_normal((200, 64)).astype(np.float32)
    b /= np.linalg.norm(b, axis=1, keepdims=True)
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    st = assert_exact(b, q, k, prec)
    assert st["n_fallback"] <= 2


def test_fp32_form_by_size():
    """FP32, up to 16 neighbours: lists for many queries over few rows, thresholds on
    the other side of each line, for real values and for exact ones (the form is read
    from the trace of a child process); the same ids from both."""
    import subprocess
    import sys
    real = [(6000, 896, 2, "topc"), (5999, 896, 2, "thresh"), (6000, 897, 4, "thresh"),
            (16384, 1024, 4, "topc"), (65536, 2048, 3, "topc"), (65536, 2049, 3, "thresh"),
            (8192, 512, 5, "topc"), (8191, 512, 5, "thresh"), (8192, 513, 8, "thresh"),
            (65536, 896, 8, "topc"), (65536, 896, 9, "thresh"), (300, 100, 2, "thresh")]
    exact = [(3000, 4096, 2, "topc"), (2999, 4096, 2, "thresh"), (3000, 4097, 2, "thresh"),
             (3000, 2048, 3, "topc"), (3000, 2049, 4, "thresh"), (6000, 1024, 5, "topc"),
             (5999, 1024, 5, "thresh"), (6000, 1025, 8, "thresh"), (6000, 512, 16, "topc"),
             (6000, 512, 17, "thresh"), (65536, 1024, 9, "topc"), (65536, 1025, 9, "thresh")]
    code = (
        "import numpy as np, sys, yael_gb300 as yg; sys.path.insert(0, 'tests')\n"
        "from _util import knn_mismatches\n"
        "rng = np.random.default_rng(7)\n"
        "for shapes, exact in ((%r, 0), (%r, 1)):\n"
        "    for nq, nb, k, form in shapes:\n"
        "        b, q = rng.standard_normal((nb, 12)), rng.standard_normal((nq, 12))\n"
        "        if exact: b, q = np.round(20 * b), np.round(20 * q)\n"
        "        b, q = b.astype(np.float32), q.astype(np.float32)\n"
        "        idx, _ = yg.knn(q, b, nnn=k, precision='fp32')\n"
        "        assert knn_mismatches(b, q, idx)[0] == 0, (nq, nb, k, exact)\n" % (real, exact))
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True,
                       env=dict(os.environ, YAEL_GPU_TRACE="1"), timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    first = [ln for ln in r.stderr.splitlines() if "knn level=0" in ln]
    assert len(first) == len(real + exact)
    for (nq, nb, k, form), ln in zip(real + exact, first):
        assert f"pass={form} nq={nq} nb={nb} " in ln, ln


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("nb", [50, 100, 128, 129, 256, 300, 512, 513, 1025])
def test_rerank_at_its_candidate_counts(nb, prec):
    """Bases in which every row, or nearly, is a candidate, at the counts where the
    re-rank changes its form: real values, integers with many ties, and integer
    rows against real queries."""
    rng = np.random.default_rng(nb)
    b = rng.standard_normal((nb, 20)).astype(np.float32)
    q = rng.standard_normal((70, 20)).astype(np.float32)
    bi, qi = np.round(b).astype(np.float32), np.round(q).astype(np.float32)
    for k in (17, 33, 50):
        assert_exact(b, q, k, prec)
        assert assert_exact(bi, qi, k, prec)["exact_class"] == 1
        assert_exact(bi, q, k, prec)


@pytest.mark.parametrize("nq,nb,d,k", [(1, 40_000, 33, 2), (3, 25_000, 16, 20), (130, 12_000, 40, 5)])
def test_fp32_sample_tiles_of_their_own(nq, nb, d, k):
    """Few queries over a base that fills the GPU with 128-row query tiles and whose
    sample does not: the sample's tiles have 32 rows."""
    rng = np.random.default_rng(nb + k)
    b = rng.standard_normal((nb, d)).astype(np.float32)
    q = rng.standard_normal((nq, d)).astype(np.float32)
    st = assert_exact(b, q, k, "fp32")
    assert st["n_fallback"] == 0
    assert_exact(np.round(4 * b).astype(np.float32), np.round(4 * q).astype(np.float32), k, "fp32")


@pytest.mark.parametrize("prec", PRECS)
@pytest.mark.parametrize("nq,nb,k", [(2000, 30_000, 300), (300, 30_000, 315), (2000, 9000, 250)])
def test_rerank_slots_of_long_lists(nq, nb, k, prec):
    """Candidate slots of 8,192 cut to 4,096 where they hold the expected candidates
    three times: exact, with next to no rejected query."""
    rng = np.random.default_rng(nb + k)
    b = rng.standard_normal((nb, 24)).astype(np.float32)
    q = rng.standard_normal((nq, 24)).astype(np.float32)
    st = assert_exact(b, q, k, prec)
    assert st["n_band"] <= 3 and st["n_fallback"] == 0
