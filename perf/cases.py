"""Performance cases of the exhaustive k-NN engine.

Each case is one call (or one request window) that a program using the
library makes: host matrices through the Python API (``searchbatch``,
``allknn``), device buffers through the C ABI (``ssg_search_device``,
``ssg_allknn_device``, ``ssg_search_batches``), and the learned shortlist's
training.  Sizes follow the benchmark's configurations (C1-C5 of
``workloads.py``) and generic ragged sizes beside them; inputs are seeded
synthetic data of the same distributions, made on the GPU.
"""
from __future__ import annotations

import ctypes as C
import importlib.util
import math
import os
import random
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    name = "similaritysearch_gb300"
    if name not in sys.modules:
        pkg_dir = os.path.join(ROOT, "similaritysearch.jl_gb300")
        spec = importlib.util.spec_from_file_location(
            name, os.path.join(pkg_dir, "__init__.py"), submodule_search_locations=[pkg_dir])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------

def _search(name, via, prec, metric, n, dim, m, k, data="mixture", elem="f32", overfetch=4.0):
    return {"name": name, "op": "search", "via": via, "prec": prec, "metric": metric, "n": n, "dim": dim, "m": m,
            "k": k, "data": data, "elem": elem, "overfetch": overfetch}


def listed():
    return [
        # one `search(index, ctx, q, res)` of an interactive program: latency
        _search("fp32_one_query", "host", "fp32", "sql2", 100_000, 128, 1, 10, data="gauss"),
        # C1: the reference's searchbatch of a thousand queries
        _search("fp32_c1", "host", "fp32", "sql2", 100_000, 128, 1000, 10, data="gauss"),
        # wide half-precision embeddings (CastF32 twin), ragged sizes, a longer list
        _search("fp32_wide_ragged", "host", "fp32", "cosine", 200_003, 300, 777, 30, elem="f16"),
        # all-vs-all neighbours of a mid-sized collection, exact, ragged sizes
        {"name": "fp32_allknn_ragged", "op": "allknn", "via": "host", "prec": "fp32", "metric": "cosine",
         "n": 100_003, "dim": 100, "k": 15, "exclude_self": 0, "data": "mixture", "overfetch": 4.0},
        # C2, the benchmark's headline: allknn over a million vectors, BF16 with exact rerank
        {"name": "bf16_allknn_c2", "op": "allknn", "via": "device", "prec": "bf16", "metric": "normcosine",
         "n": 1_000_000, "dim": 96, "k": 32, "exclude_self": 1, "data": "mixture", "overfetch": 1.5},
        # an ordinary batch against the same collection
        _search("bf16_batch", "device", "bf16", "normcosine", 1_000_000, 96, 2048, 10, overfetch=2.0),
        # C4: one median request of the stream, squared distances at the calibrated over-fetch
        _search("fp8_request", "device", "fp8", "sql2", 2_000_000, 768, 64, 10, overfetch=12.0),
        # C4: the stream's largest request, inner products, long lists
        _search("fp8_large_request", "device", "fp8", "ip", 2_000_000, 768, 4096, 100, overfetch=1.25),
        # C4: a window of eight coalesced requests of uneven size and k
        {"name": "fp8_window", "op": "batches", "via": "device", "prec": "fp8", "metric": "ip", "n": 2_000_000,
         "dim": 768, "nb": 8, "sizes": 13, "data": "mixture", "overfetch": 1.25},
        # C3: ten thousand sketch queries, and one request's worth of them
        _search("hamming_c3", "device", "fp32", "hamming", 2_000_000, 16, 10_000, 100, data="bits"),
        _search("hamming_request", "device", "fp32", "hamming", 2_000_000, 16, 64, 100, data="bits"),
        # C5 in small: train the shortlist network, embed the database, search through it
        {"name": "learned_train_search", "op": "train", "via": "device", "prec": "fp32", "metric": "sql2",
         "n": 200_000, "dim": 768, "m": 1000, "k": 10, "sample": 20_000, "triplets": 200_000, "hidden": 256,
         "out_dim": 64, "batch": 1024, "data": "mixture"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["fp32", "fp32", "allknn", "bf16", "fp8", "batches", "hamming", "hamming"])
    if kind == "fp32":
        elem = rng.choice(["f32", "f32", "f16", "u8"])
        c = _search("", rng.choice(["host", "device"]), "fp32", rng.choice(["sql2", "l2", "cosine", "normcosine"]),
                    _log(rng, 10_000, 300_000), _log(rng, 16, 768), _log(rng, 1, 1000), _log(rng, 1, 100),
                    data=rng.choice(["gauss", "mixture"]), elem=elem)
        if elem == "u8" and c["metric"] == "normcosine":
            c["metric"] = "cosine"
    elif kind == "allknn":
        prec = rng.choice(["fp32", "bf16"])
        c = {"op": "allknn", "via": rng.choice(["host", "device"]), "prec": prec,
             "metric": rng.choice(["sql2", "l2", "cosine", "normcosine"]),
             "n": _log(rng, 5_000, 150_000 if prec == "fp32" else 400_000), "dim": _log(rng, 16, 128),
             "k": rng.randint(2, 40), "exclude_self": 0, "data": "mixture", "overfetch": rng.choice([1.5, 2.0, 4.0])}
    elif kind == "bf16":
        c = _search("", "device", "bf16", rng.choice(["sql2", "cosine", "normcosine"]), _log(rng, 20_000, 1_000_000),
                    _log(rng, 32, 256), _log(rng, 1, 4096), rng.randint(1, 20), overfetch=rng.choice([1.5, 2.0, 4.0]))
    elif kind == "fp8":
        c = _search("", "device", "fp8", rng.choice(["sql2", "ip", "cosine"]), _log(rng, 100_000, 2_000_000),
                    _log(rng, 64, 768), _log(rng, 1, 4096), rng.choice([1, 10, 100]), overfetch=1.25)
        if c["k"] <= 10:
            c["overfetch"] = rng.choice([1.25, 4.0, 12.0])
    elif kind == "batches":
        c = {"op": "batches", "via": "device", "prec": "fp8", "metric": rng.choice(["ip", "sql2"]),
             "n": _log(rng, 200_000, 2_000_000), "dim": rng.randint(64, 768), "nb": rng.randint(2, 8),
             "sizes": rng.randrange(1 << 20), "data": "mixture", "overfetch": 1.25}
    else:
        c = _search("", "device", "fp32", "hamming", _log(rng, 50_000, 2_000_000), _log(rng, 1, 16),
                    _log(rng, 1, 10_000), _log(rng, 1, 100), data="bits")
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _mixture(g, count, dim, unit, centres=None):
    """Rows of a Gaussian mixture (centres N(0, 1), per-cluster sigma), made
    unit length; log-normal norms unless `unit`."""
    if centres is None:
        kc = 1000 if dim <= 128 else 4096
        centres = (torch.randn(kc, dim, generator=g, device="cuda"),
                   torch.rand(kc, generator=g, device="cuda") * 0.4 + 0.1)
    cen, sig = centres
    out = torch.empty(count, dim, device="cuda")
    for s in range(0, count, 250_000):
        c = min(250_000, count - s)
        lab = torch.randint(0, cen.shape[0], (c,), generator=g, device="cuda")
        blk = torch.randn(c, dim, generator=g, device="cuda") * sig[lab, None] + cen[lab]
        blk /= blk.norm(dim=1, keepdim=True)
        if not unit:
            blk *= torch.exp(0.25 * torch.randn(c, 1, generator=g, device="cuda"))
        out[s:s + c] = blk
    return out, centres


def _sizes(case):
    """Request sizes and k of a window of the stream (at most 1,024 queries each)."""
    r = np.random.default_rng(case["sizes"])
    sizes = np.clip(np.round(r.lognormal(np.log(64), 1.0, size=case["nb"])), 1, 1024).astype(int)
    ks = [(1, 10, 100)[i % 3] for i in range(case["nb"])]
    return sizes.tolist(), ks


def _inputs(case, seed):
    """(database (n, dim), queries (m, dim)) as CUDA tensors; queries are None for allknn."""
    g = torch.Generator(device="cuda")
    g.manual_seed(1_000_003 * (seed + 1) + 17)
    n, dim = case["n"], case["dim"]
    m = sum(_sizes(case)[0]) if case["op"] == "batches" else case.get("m", 0)
    if case["data"] == "bits":
        x = torch.randint(-2**63, 2**63 - 1, (n, dim), generator=g, device="cuda", dtype=torch.int64)
        src = torch.randint(0, n, (m,), generator=g, device="cuda")
        # each query: a database sketch with every bit flipped with probability 0.1
        w = torch.ones(64, dtype=torch.int64, device="cuda") << torch.arange(64, device="cuda")
        q = torch.empty(m, dim, dtype=torch.int64, device="cuda")
        for s in range(0, m, 1024):
            e = min(m, s + 1024)
            flips = torch.rand(e - s, dim, 64, generator=g, device="cuda") < 0.1
            q[s:e] = x[src[s:e]] ^ (flips.to(torch.int64) * w).sum(dim=2)
        return x, q
    unit = case["metric"] == "normcosine"
    if case["data"] == "gauss":
        x = torch.randn(n, dim, generator=g, device="cuda")
        q = torch.randn(m, dim, generator=g, device="cuda") if m else None
        if unit:
            x /= x.norm(dim=1, keepdim=True)
            if m:
                q /= q.norm(dim=1, keepdim=True)
    else:
        x, cen = _mixture(g, n, dim, unit)
        q = _mixture(g, m, dim, unit, cen)[0] if m else None
    elem = case.get("elem", "f32")
    if elem == "f16":
        x, q = x.half(), q.half()
    elif elem == "u8":
        scale = 20.0 if case["data"] == "gauss" else 20.0 * math.sqrt(dim)
        x, q = ((t * scale + 128).clamp(0, 255).to(torch.uint8) for t in (x, q))
    return x, q


# ---------------------------------------------------------------------------
# Preparation and the pass
# ---------------------------------------------------------------------------

def _dist(ss, metric, cast):
    D = ss.Dist.CastF32 if cast else ss.Dist
    return {"sql2": D.SqL2, "l2": D.L2, "cosine": D.Cosine, "normcosine": D.NormCosine}[metric]()


class _Index:
    """An index over a device database through the C ABI, on torch's stream."""

    def __init__(self, ss, case, x):
        N = ss._native
        self.N, self.L = N, N.lib()
        metric = {"sql2": N.METRIC_SQL2, "l2": N.METRIC_L2, "normcosine": N.METRIC_NORMCOSINE,
                  "cosine": N.METRIC_COSINE, "ip": N.METRIC_IP, "hamming": N.METRIC_HAMMING}[case["metric"]]
        elem = {torch.float32: N.ELEM_F32, torch.float16: N.ELEM_F16, torch.uint8: N.ELEM_U8,
                torch.int64: N.ELEM_U64}[x.dtype]
        prec = {"fp32": N.PREC_FP32, "bf16": N.PREC_BF16, "fp8": N.PREC_FP8}[case["prec"]]
        torch.cuda.synchronize()
        h = C.c_void_p()
        N.check(self.L.ssg_create_device(metric, elem, x.shape[1], x.shape[0], C.c_void_p(x.data_ptr()), x.shape[1],
                                         prec, C.byref(h)))
        self.h = h
        self.call("ssg_set_stream", C.c_void_p(torch.cuda.current_stream().cuda_stream))
        if case["prec"] != "fp32":
            self.call("ssg_set_param", b"overfetch", float(case["overfetch"]))

    def call(self, name, *args):
        self.N.check(getattr(self.L, name)(self.h, *args), self.h)

    def __del__(self):
        if getattr(self, "h", None):
            self.L.ssg_destroy(self.h)


def prepare(case, seed):
    ss = _package()
    x, q = _inputs(case, seed)
    if case["via"] == "host":
        cast = case.get("elem", "f32") != "f32"
        idx = ss.GPUExhaustiveSearch(_dist(ss, case["metric"], cast), ss.MatrixDatabase.from_rows(x.cpu().numpy()),
                                     precision=case["prec"])
        if case["prec"] != "fp32":
            idx.set_param("overfetch", case["overfetch"])
        Q = None if q is None else ss.MatrixDatabase.from_rows(q.cpu().numpy())
        return {"case": case, "ss": ss, "idx": idx, "ctx": ss.GenericContext(logger=None), "Q": Q}
    st = {"case": case, "ss": ss, "idx": _Index(ss, case, x), "q": q}
    if case["op"] == "batches":
        sizes, ks = _sizes(case)
        st["sizes"], st["ks"] = sizes, ks
        st["parts"] = list(torch.split(q, sizes))
    if case["op"] == "train":
        st["dir"] = tempfile.TemporaryDirectory()
        st["path"] = os.path.join(st["dir"].name, "model.bin")
        st["seed"] = seed + 15
        st["idx"].call("ssg_set_param", b"learned_target", 0.0)
    return st


def _outputs(m, k):
    return (torch.empty(m, k, dtype=torch.int32, device="cuda"), torch.empty(m, k, dtype=torch.float32, device="cuda"))


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def run(state):
    case, ss, idx = state["case"], state["ss"], state["idx"]
    if case["via"] == "host":
        if case["op"] == "allknn":
            ids, dists = ss.allknn(idx, state["ctx"], case["k"], exclude_self=bool(case["exclude_self"]))
        else:
            ids, dists = ss.searchbatch(idx, state["ctx"], state["Q"], case["k"])
        return {"ids": ids.T.view(np.int32), "dists": dists.T}
    if case["op"] == "allknn":
        ids, dists = _outputs(case["n"], case["k"])
        idx.call("ssg_allknn_device", case["k"], case["exclude_self"], _ptr(ids), _ptr(dists))
        return {"ids": ids, "dists": dists}
    if case["op"] == "batches":
        sizes, ks, parts = state["sizes"], state["ks"], state["parts"]
        outs = [_outputs(m, k) for m, k in zip(sizes, ks)]
        nb = len(sizes)
        P = C.c_void_p * nb
        idx.call("ssg_search_batches", nb, P(*[p.data_ptr() for p in parts]), (C.c_int64 * nb)(*sizes),
                 (C.c_int32 * nb)(*ks), P(*[i.data_ptr() for i, _ in outs]), P(*[d.data_ptr() for _, d in outs]))
        return {"ids": [i for i, _ in outs], "dists": [d for _, d in outs]}
    res = {}
    if case["op"] == "train":
        idx.call("ssg_train_mlp", case["sample"], case["triplets"], 1, case["hidden"], case["out_dim"], case["batch"],
                 1e-3, state["seed"])
        idx.call("ssg_save_model", state["path"].encode())
        # 8-byte magic and three int64 sizes, then the FP32 weights
        res["weights"] = np.fromfile(state["path"], dtype=np.float32, offset=32)
    ids, dists = _outputs(case["m"], case["k"])
    idx.call("ssg_search_device", _ptr(state["q"]), case["m"], case["k"], _ptr(ids), _ptr(dists), 0)
    res["ids"], res["dists"] = ids, dists
    return res


# ---------------------------------------------------------------------------
# What a pass cannot do without, and its 64-bit results
# ---------------------------------------------------------------------------

def work(case):
    """The database once in the form the method scans (FP32, BF16, FP8,
    sketch words), the queries and the results once; two operations per
    element (per bit for sketches) and pair."""
    n, dim = case["n"], case["dim"]
    es = 8 if case["metric"] == "hamming" else {"fp32": 4, "bf16": 2, "fp8": 1}[case["prec"]]
    per = 128 if case["metric"] == "hamming" else 2
    if case["op"] == "allknn":
        return {"bytes": n * dim * es + n * case["k"] * 8, "flops": per * n * n * dim}
    if case["op"] == "batches":
        sizes, ks = _sizes(case)
        m, res = sum(sizes), sum(a * b for a, b in zip(sizes, ks))
        return {"bytes": n * dim * es + m * dim * 4 + res * 8, "flops": per * m * n * dim}
    m, k = case["m"], case["k"]
    if case["op"] == "train":
        # forward and backward of every triplet's three rows, the database's
        # embedding, the sample's neighbours, the shortlist's scan
        net = case["dim"] * case["hidden"] + case["hidden"] * case["out_dim"]
        flops = 6 * 3 * case["triplets"] * net + 2 * n * net + 2 * case["sample"] ** 2 * dim \
            + 2 * m * (net + n * case["out_dim"])
        return {"bytes": n * dim * 4 + 3 * case["triplets"] * dim * 4 + n * case["out_dim"] * 2 + m * k * 8,
                "flops": flops}
    qe = 8 if case["metric"] == "hamming" else 4
    return {"bytes": n * dim * es + m * dim * qe + m * k * 8, "flops": per * m * n * dim}


def _bits(x):
    """Sketch words -> +-1 per bit (Float32)."""
    b = (x[:, :, None] >> torch.arange(64, device=x.device)) & 1
    return (1 - 2 * b).reshape(x.shape[0], -1).float()


def _exact_float(metric, x, q, k, drop_self, q0):
    """The k smallest distances of each query in 64 bits: an FP32 shortlist,
    its distances in Float64."""
    kk = min(x.shape[0], k + drop_self + 32)
    xf, qf = x.float(), q.float()
    best_v = best_i = None
    for s in range(0, xf.shape[0], 100_000):
        xs = xf[s:s + 100_000]
        v = -(qf @ xs.T)
        if metric in ("sql2", "l2"):
            v = (xs * xs).sum(1) + 2 * v
        elif metric == "cosine":
            v = v / xs.norm(dim=1)
        v, i = torch.topk(v, min(kk, v.shape[1]), dim=1, largest=False)
        i = i + s
        if best_v is not None:
            v, i = torch.cat([best_v, v], 1), torch.cat([best_i, i], 1)
            v, j = torch.topk(v, min(kk, v.shape[1]), dim=1, largest=False)
            i = torch.gather(i, 1, j)
        best_v, best_i = v, i
    out = []
    for s in range(0, qf.shape[0], 512):
        qs, ids = q[s:s + 512].double(), best_i[s:s + 512]
        c = x[ids].double()
        if metric in ("sql2", "l2"):
            d = ((c - qs[:, None]) ** 2).sum(2)
            d = d.sqrt() if metric == "l2" else d
        else:
            d = -(c * qs[:, None]).sum(2)
            if metric == "cosine":
                d = 1 + d / (c.norm(dim=2) * qs.norm(dim=1, keepdim=True))
            elif metric == "normcosine":
                d = 1 + d
        if drop_self:
            me = torch.arange(q0 + s, q0 + s + qs.shape[0], device=d.device)[:, None]
            d = torch.where(ids == me, torch.full_like(d, math.inf), d)
        out.append(d.sort(dim=1).values[:, :k])
    return torch.cat(out)


def _exact_hamming(x, q, k):
    qb, bits, best = _bits(q), x.shape[1] * 64, None
    for s in range(0, x.shape[0], 50_000):
        v = torch.topk(qb @ _bits(x[s:s + 50_000]).T, min(k, x.shape[0] - s, 50_000), dim=1).values
        best = v if best is None else torch.topk(torch.cat([best, v], 1), min(k, best.shape[1] + v.shape[1]), dim=1).values
    return ((bits - best) / 2).double()


def exact(case, seed):
    if case["op"] == "train":
        return None
    m = case["n"] if case["op"] == "allknn" else sum(_sizes(case)[0]) if case["op"] == "batches" else case["m"]
    if m * case["n"] > 1e11:
        return None
    x, q = _inputs(case, seed)
    if case["metric"] == "hamming":
        d = torch.cat([_exact_hamming(x, c, case["k"]) for c in torch.split(q, 4096)])
        return {"ids": None, "dists": d}
    if case["op"] == "batches":
        sizes, ks = _sizes(case)
        return {"ids": [None] * len(sizes),
                "dists": [_exact_float(case["metric"], x, c, k, 0, 0) for c, k in zip(torch.split(q, sizes), ks)]}
    q, drop = (x, case["exclude_self"]) if q is None else (q, 0)
    d = torch.cat([_exact_float(case["metric"], x, c, case["k"], drop, 4096 * i)
                   for i, c in enumerate(torch.split(q, 4096))])
    return {"ids": None, "dists": d}
