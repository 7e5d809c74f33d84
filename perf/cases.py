"""The calls whose speed this repository is measured by: exact k-NN, k-means,
hierarchical k-means, Gaussian mixtures, Fisher vectors and VLAD through their
public entry points, from one query to the large configurations.

A case is a dict of plain values; ``family`` names the call and the rest are
its sizes and options.  Device-resident callers use the extension API with
device pointers (``yael_gpu_knn_ex`` and relatives), the descriptor and mixture
calls take numpy arrays through the package's front end, as their users do.
"""
import ctypes
import math
import os
import random

import numpy as np
import torch

import yael_gb300 as yg

PREC = {"fp32": yg.PREC_FP32, "bf16": yg.PREC_BF16, "fp16": yg.PREC_FP16}


def listed():
    return [
        # one query against a small base, FP32 (the default): an interactive
        # search, where launches and round trips are all there is
        {"name": "knn_one_query", "family": "knn", "nq": 1, "nb": 10_000, "d": 128, "k": 10,
         "prec": "fp32", "metric": 2, "data": "sift"},
        # a batch of real-valued queries in the default precision, ragged sizes
        {"name": "knn_fp32", "family": "knn", "nq": 1000, "nb": 100_003, "d": 100, "k": 20,
         "prec": "fp32", "metric": 2, "data": "unit"},
        # the headline: SIFT-like descriptors, 100 neighbours among a million
        {"name": "knn_bf16", "family": "knn", "nq": 10_000, "nb": 1_000_000, "d": 128, "k": 100,
         "prec": "bf16", "metric": 2, "data": "sift"},
        # vector quantisation: the nearest of many centroids for each descriptor
        {"name": "quantise", "family": "knn", "nq": 200_003, "nb": 10_000, "d": 128, "k": 1,
         "prec": "bf16", "metric": 2, "data": "mixture"},
        # many independent searches of uneven sizes in one call (inverted lists)
        {"name": "knn_batch", "family": "knn_batch", "pairs": 64, "nq_max": 8192,
         "nb_max": 1_000_000, "d": 128, "k": 32, "metric": 2},
        # a small vocabulary on the tensor cores: the small k-means configuration
        {"name": "kmeans_k256", "family": "kmeans", "n": 100_000, "d": 128, "k": 256, "niter": 20,
         "prec": "bf16"},
        # a large vocabulary: the large configuration with a fifth of its points
        {"name": "kmeans_k16384", "family": "kmeans", "n": 2_000_000, "d": 128, "k": 16_384,
         "niter": 5, "prec": "bf16"},
        # what the drop-in k-means runs by default: FP32, a hundred clusters
        {"name": "kmeans_fp32", "family": "kmeans", "n": 50_000, "d": 64, "k": 100, "niter": 30,
         "prec": "fp32"},
        # a vocabulary tree from host memory: the tree configuration on half its points
        {"name": "hkm_tree", "family": "hkm", "n": 1_000_000, "d": 96, "bf": 32, "nlevel": 3,
         "niter": 15, "prec": "bf16"},
        # learning the mixture of a Fisher-vector pipeline from host memory
        {"name": "gmm_learn", "family": "gmm_learn", "n": 100_000, "d": 128, "k": 256,
         "niter": 10},
        # one image's Fisher vector: a few thousand reduced descriptors
        {"name": "fisher", "family": "fisher", "n": 2000, "d": 64, "k": 256},
        # one image's VLAD descriptor
        {"name": "vlad", "family": "vlad", "n": 2000, "d": 128, "k": 64},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random):
    """One more case: a family, then its sizes over their whole range."""
    family = rng.choice(["knn", "knn", "knn_batch", "kmeans", "kmeans", "hkm", "gmm_learn",
                         "fisher", "vlad"])
    if family == "knn":
        prec = rng.choice(["fp32", "fp32", "bf16", "bf16", "fp16"])
        d = rng.choice([32, 64, 96, 100, 128, rng.randint(17, 200)])
        nq = _log_int(rng, 1, 200_000)
        nb = _log_int(rng, 2000, 1_000_000)
        # no search costs more than the largest listed cases
        most = 6.4e10 if prec == "fp32" else 2.5e12
        while 2.0 * nq * nb * d > most:
            nq, nb = max(1, int(nq * 0.61)), max(2000, int(nb * 0.83))
        k = rng.choice([1, 1, 2, 5, 10, 20, 50, 100])
        # inner products of unit vectors, distances of everything
        data = rng.choice(["sift", "unit", "mixture"])
        # fp16 operands hold squared norms below 2^15, SIFT's are above it
        if prec == "fp16" and data == "sift":
            data = "unit"
        metric = 16 if data == "unit" and rng.random() < 0.4 else 2
        return {"family": family, "nq": nq, "nb": nb, "d": d, "k": k, "prec": prec,
                "metric": metric, "data": data}
    if family == "knn_batch":
        return {"family": family, "pairs": rng.randint(4, 64),
                "nq_max": _log_int(rng, 64, 8192), "nb_max": _log_int(rng, 20_000, 1_000_000),
                "d": rng.choice([64, 96, 128]), "k": rng.choice([10, 16, 32, 50]),
                "metric": rng.choice([2, 2, 16])}
    if family == "kmeans":
        prec = rng.choice(["fp32", "bf16", "bf16"])
        d = rng.choice([32, 64, 96, 128, rng.randint(17, 160)])
        n = _log_int(rng, 5000, 1_000_000)
        k = _log_int(rng, 8, min(16_384, n // 30))
        niter = rng.randint(3, 20)
        most = 2e11 if prec == "fp32" else 1e13
        while 2.0 * n * k * d * niter > most:
            if niter > 5:
                niter -= 1
            else:
                k = max(8, int(k * 0.8))
                n = max(30 * k, int(n * 0.9))
        return {"family": family, "n": n, "d": d, "k": k, "niter": niter, "prec": prec}
    if family == "hkm":
        bf = rng.choice([8, 10, 16, 32])
        nlevel = rng.choice([2, 3])
        n = _log_int(rng, 20_000, 600_000)
        n = max(n, 30 * bf ** nlevel)
        return {"family": family, "n": n, "d": rng.choice([32, 64, 96, 128]), "bf": bf,
                "nlevel": nlevel, "niter": rng.randint(5, 15),
                "prec": rng.choice(["fp32", "bf16", "bf16"])}
    if family == "gmm_learn":
        return {"family": family, "n": _log_int(rng, 5000, 100_000),
                "d": rng.choice([32, 64, 100, 128, rng.randint(20, 128)]),
                "k": rng.choice([16, 64, 100, 128, 256]), "niter": rng.randint(4, 10)}
    if family == "fisher":
        return {"family": family, "n": _log_int(rng, 200, 100_000),
                "d": rng.choice([32, 64, 100, 128, rng.randint(20, 128)]),
                "k": rng.choice([16, 64, 100, 256])}
    return {"family": "vlad", "n": _log_int(rng, 200, 200_000),
            "d": rng.choice([32, 64, 96, 128, rng.randint(20, 128)]),
            "k": rng.choice([16, 64, 100, 256])}


# ---------------------------------------------------------------------------
# inputs


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _sift(n, d, g):
    """SIFT-like integer descriptors: 30% zeros, else floor|N(0, 40)| up to 255."""
    v = (torch.randn((n, d), device="cuda", generator=g).abs_() * 40.0).floor_().clamp_(max=255.0)
    v[torch.rand((n, d), device="cuda", generator=g) < 0.3] = 0.0
    return v


def _unit(n, d, g):
    v = torch.randn((n, d), device="cuda", generator=g)
    return v / v.norm(dim=1, keepdim=True)


def _mixture(n, centres, sigma, g):
    lab = torch.randint(0, centres.shape[0], (n,), device="cuda", generator=g)
    return centres[lab] + sigma * torch.randn((n, centres.shape[1]), device="cuda", generator=g)


def _search_data(case, nq, nb, g):
    """Queries and base of one search."""
    d = case["d"]
    if case["data"] == "sift":
        return _sift(nq, d, g), _sift(nb, d, g)
    if case["data"] == "unit":
        return _unit(nq, d, g), _unit(nb, d, g)
    # descriptors around the words of a vocabulary, which is the base
    words = torch.randn((nb, d), device="cuda", generator=g)
    return _mixture(nq, words, 0.2, g), words


def _batch_sizes(case):
    """Pair sizes, log-uniform; they belong to the case, not to the seed."""
    rng = random.Random(case["pairs"] * 1_000_003 + case["nq_max"])
    return [(_log_int(rng, 1, case["nq_max"]), _log_int(rng, 10_000, case["nb_max"]))
            for _ in range(case["pairs"])]


def _mixture_model(case, g):
    """(w, mu, sigma) of a mixture such as gmm_learn gives, as host arrays."""
    k, d = case["k"], case["d"]
    w = torch.rand(k, device="cuda", generator=g) + 0.5
    mu = torch.randn((k, d), device="cuda", generator=g)
    sigma = 0.25 * (torch.rand((k, d), device="cuda", generator=g) + 0.5)
    return tuple(x.float().cpu().numpy() for x in (w / w.sum(), mu, sigma))


class State:
    """What a user's program holds: the inputs, and buffers for the outputs."""

    def __init__(self, case):
        self.case = case


def _host(t):
    return t.float().cpu().numpy()


def prepare(case, seed):
    g = _generator(seed)
    s = State(case)
    family = case["family"]
    if family == "knn":
        s.q, s.b = _search_data(case, case["nq"], case["nb"], g)
        s.idx = torch.empty((case["nq"], case["k"]), dtype=torch.int32, device="cuda")
        s.dis = torch.empty((case["nq"], case["k"]), dtype=torch.float32, device="cuda")
    elif family == "knn_batch":
        sizes = _batch_sizes(case)
        s.pairs = [(_unit(nq, case["d"], g), _unit(nb, case["d"], g)) for nq, nb in sizes]
        # the results of all the pairs, one pair after the other
        rows = sum(nq for nq, _ in sizes)
        s.idx = torch.empty((rows, case["k"]), dtype=torch.int32, device="cuda")
        s.dis = torch.empty((rows, case["k"]), dtype=torch.float32, device="cuda")
    elif family == "kmeans":
        comps = min(case["k"], 65_536)
        centres = torch.randn((comps, case["d"]), device="cuda", generator=g)
        s.v = _mixture(case["n"], centres, 0.15, g)
        s.centroids = torch.empty((case["k"], case["d"]), dtype=torch.float32, device="cuda")
        s.dis = torch.empty(case["n"], dtype=torch.float32, device="cuda")
        s.assign = torch.empty(case["n"], dtype=torch.int32, device="cuda")
        s.nassign = torch.empty(case["k"], dtype=torch.int32, device="cuda")
    elif family == "hkm":
        centres = torch.randn((4096, case["d"]), device="cuda", generator=g)
        v = _mixture(case["n"], centres, 0.1, g)
        # page-locked, as a program that streams its descriptors to the GPU holds them
        s.v = torch.empty(v.shape, dtype=torch.float32, pin_memory=True)
        s.v.copy_(v)
        rows = sum(case["bf"] ** (level + 1) for level in range(case["nlevel"]))
        s.centroids = np.empty((rows, case["d"]), dtype=np.float32)
        s.assign = np.empty(case["n"], dtype=np.int32)
    elif family == "gmm_learn":
        centres = torch.randn((case["k"], case["d"]), device="cuda", generator=g)
        s.v = _host(_mixture(case["n"], centres, 0.5, g))
    elif family == "fisher":
        s.model = _mixture_model(case, g)
        s.v = _host(_mixture(case["n"], torch.from_numpy(s.model[1]).cuda(), 0.6, g))
    elif family == "vlad":
        s.c = _host(_sift(case["k"], case["d"], g))
        s.v = _host(_sift(case["n"], case["d"], g))
    else:
        raise ValueError(f"unknown family {family}")
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------------------
# one pass


def _precision(name):
    """The calls without a precision argument read it from the environment."""
    os.environ["YAEL_GPU_PRECISION"] = name


def _check(rc):
    if rc != 0:
        raise RuntimeError(f"call failed ({rc}): {yg.last_error()}")


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


_libc = ctypes.CDLL(None)
_libc.srand48.argtypes = [ctypes.c_long]


def run(state):
    case = state.case
    family = case["family"]
    L = yg.lib()
    if family == "knn":
        opts = yg.KnnOpts(PREC[case["prec"]], case["metric"], 1, _stream())
        _check(L.yael_gpu_knn_ex(case["nq"], case["nb"], case["d"], case["k"], state.b.data_ptr(),
                                 state.q.data_ptr(), state.idx.data_ptr(), state.dis.data_ptr(),
                                 ctypes.byref(opts)))
        return state.idx, state.dis
    if family == "knn_batch":
        pairs = (yg.KnnPair * len(state.pairs))()
        idx, dis, pitch = state.idx.data_ptr(), state.dis.data_ptr(), 4 * case["k"]
        row = 0
        for i, (q, b) in enumerate(state.pairs):
            pairs[i] = yg.KnnPair(q.shape[0], b.shape[0], q.data_ptr(), b.data_ptr(),
                                  idx + row * pitch, dis + row * pitch)
            row += q.shape[0]
        opts = yg.KnnOpts(yg.PREC_BF16, case["metric"], 1, _stream())
        _check(L.yael_gpu_knn_batch(len(state.pairs), ctypes.cast(pairs, ctypes.c_void_p),
                                    case["d"], case["k"], ctypes.byref(opts)))
        return state.idx, state.dis
    if family == "kmeans":
        opts = yg.KmeansOpts(PREC[case["prec"]], 1, _stream())
        flags = yg.KMEANS_QUIET | yg.KMEANS_INIT_RANDOM
        qerr = L.yael_gpu_kmeans_ex(case["d"], case["n"], case["k"], case["niter"],
                                    state.v.data_ptr(), flags, 1234, 1,
                                    state.centroids.data_ptr(), state.dis.data_ptr(),
                                    state.assign.data_ptr(), state.nassign.data_ptr(),
                                    ctypes.byref(opts))
        _check(opts.status)
        return state.centroids, state.dis, state.assign, state.nassign, float(qerr)
    if family == "hkm":
        _precision(case["prec"])
        _libc.srand48(1234)  # the seeds of the nodes come from lrand48()
        _check(L.yael_gpu_hkm_learn_ex(case["n"], case["d"], case["nlevel"], case["bf"],
                                       state.v.data_ptr(), case["niter"], 1,
                                       state.centroids.ctypes.data, state.assign.ctypes.data,
                                       None, None))
        return state.centroids, state.assign
    _precision("fp32")
    if family == "gmm_learn":
        return yg.gmm_learn(state.v, case["k"], niter=case["niter"], seed=1234)
    if family == "fisher":
        return yg.fisher(state.model, state.v, include=("mu", "sigma"))
    return yg.vlad(state.c, state.v)


# ---------------------------------------------------------------------------
# what a pass cannot do without


def _search_work(nq, nb, d, k):
    return 4.0 * (nq + nb) * d + 8.0 * nq * k, 2.0 * nq * nb * d


def work(case):
    family = case["family"]
    if family == "knn":
        b, f = _search_work(case["nq"], case["nb"], case["d"], case["k"])
    elif family == "knn_batch":
        both = [_search_work(nq, nb, case["d"], case["k"]) for nq, nb in _batch_sizes(case)]
        b, f = sum(x[0] for x in both), sum(x[1] for x in both)
    elif family == "kmeans":
        n, d, k = case["n"], case["d"], case["k"]
        b, f = 4.0 * n * d + 8.0 * n + 4.0 * k * (d + 1), 2.0 * n * k * d * case["niter"]
    elif family == "hkm":
        n, d, bf, levels = case["n"], case["d"], case["bf"], case["nlevel"]
        b = 4.0 * n * d + 4.0 * n + 4.0 * d * sum(bf ** (i + 1) for i in range(levels))
        f = 2.0 * n * bf * d * levels * case["niter"]
    elif family == "gmm_learn":
        n, d, k = case["n"], case["d"], case["k"]
        # per iteration: three operations of a distance term, four of the two moments
        b, f = 4.0 * n * d + 4.0 * k * (2 * d + 1), 7.0 * n * k * d * case["niter"]
    elif family == "fisher":
        n, d, k = case["n"], case["d"], case["k"]
        b, f = 4.0 * n * d + 4.0 * k * (4 * d + 1), 7.0 * n * k * d
    else:
        n, d, k = case["n"], case["d"], case["k"]
        b, f = 4.0 * (n + 2 * k) * d, 2.0 * n * k * d
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the same in 64 bits


def _exact_distances(q, b, k, metric):
    """The k smallest squared distances (inner products) of each query, ascending."""
    b = b.double()
    bn = (b * b).sum(1)
    out = torch.empty((q.shape[0], k), dtype=torch.float64, device=q.device)
    step = max(1, min(q.shape[0], (1 << 28) // b.shape[0]))
    for i in range(0, q.shape[0], step):
        x = q[i:i + step].double()
        v = x @ b.t()
        if metric != 16:
            v = ((x * x).sum(1, keepdim=True) + bn) - 2.0 * v
        out[i:i + step] = v.topk(k, dim=1, largest=False, sorted=True).values
    return out


def _exact_fisher(v, model):
    w, mu, sigma = (torch.from_numpy(a).cuda().double() for a in model)
    v = torch.from_numpy(v).cuda().double()
    n, d = v.shape
    inv = 1.0 / sigma
    m = (v * v) @ inv.t() - 2.0 * (v @ (mu * inv).t()) + (mu * mu * inv).sum(1)
    x = w.log() - 0.5 * (d * math.log(2.0 * math.pi) + sigma.log().sum(1) + m)
    x = x - x.max(1, keepdim=True).values
    # densities below 2^-24 of the largest are left out
    e = torch.where(x >= -16.636, x.exp(), torch.zeros_like(x))
    p = e / e.sum(1, keepdim=True)
    s0, s1, s2 = p.sum(0)[:, None], p.t() @ v, p.t() @ (v * v)
    g_mu = (s1 - mu * s0) / sigma / (n * w[:, None] / sigma).sqrt()
    dev = s2 - 2.0 * mu * s1 + mu * mu * s0
    g_sigma = (dev / sigma - s0) / sigma.sqrt() / (2.0 * n * w[:, None] / sigma).sqrt()
    return torch.cat([g_mu.reshape(-1), g_sigma.reshape(-1)]).cpu().numpy()


def _exact_vlad(c, v):
    c, v = torch.from_numpy(c).cuda().double(), torch.from_numpy(v).cuda().double()
    out = torch.zeros_like(c)
    # integer descriptors: the distances are exact, so the first minimum is the assignment
    dis = (v * v).sum(1, keepdim=True) + (c * c).sum(1) - 2.0 * (v @ c.t())
    a = dis.min(1, keepdim=True).values
    a = (dis == a).double().argmax(1)
    out.index_add_(0, a, v - c[a])
    return out.cpu().numpy()


def exact(case, seed):
    """The outputs in 64 bits; ids have no such value.  k-means, the tree and
    the mixture start from the library's own random draws and round their
    centroids to 32 bits between iterations, so a run in 64 bits is another
    run: they have none."""
    family = case["family"]
    if family in ("kmeans", "hkm", "gmm_learn"):
        return None
    s = prepare(case, seed)
    if family == "knn":
        return None, _exact_distances(s.q, s.b, case["k"], case["metric"])
    if family == "knn_batch":
        return None, torch.cat([_exact_distances(q, b, case["k"], case["metric"])
                                for q, b in s.pairs])
    if family == "fisher":
        return _exact_fisher(s.v, s.model)
    return _exact_vlad(s.c, s.v)
