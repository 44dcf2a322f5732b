"""The seed's group minima by the rows' places in their atoms: exactly as many
keys within the bound as are wanted where the nearest rows lie in as many
groups, and databases of zero rows, whose equal distances fill every list."""
import math

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 5, 40, 150])
@pytest.mark.parametrize("m", [1, 40, 300])
def test_nearest_rows_in_as_many_groups(ss, k, m):
    rng = np.random.default_rng(k + m)
    tiles, words = 87, 4
    X = rng.integers(0, 2**64 - 1, size=(tiles * 240, words), dtype=np.uint64, endpoint=True)
    base = rng.integers(0, 2**64 - 1, size=words, dtype=np.uint64, endpoint=True)
    per = 64 if 8 * (tiles // 4) < 4 * k else 8
    samples = max(-(-4 * k // per), tiles // (12 if m <= 256 else 6))
    if 2 * samples >= 4 * k and samples >= 4:
        per = 2
    stride = max(1, int(0.618034 * samples))
    while math.gcd(stride, samples) != 1:
        stride += 1
    q = 2 * tiles // 15  # tiles between a unit's 15 atoms of 8 rows

    def row(w, c):  # column c of the w-th wide tile that the seed visits
        e = (w * stride % samples + c // 120 * samples) * 15 * q // (2 * samples)
        c %= 120
        return (e // 15 + c // 8 * q) * 120 + e % 15 * 8 + c % 8

    # a column of every group: both warps' first chunks, four places (of four
    # tiles together, or each tile's), or all eight of every chunk
    if per == 2:
        places = [row(w, 32 * seg + w % 4) for w in range(samples) for seg in range(2)]
    elif per == 8:
        places = [row(w, 32 * seg + p) for w in range(samples) for seg in range(2) for p in range(4)]
    else:
        places = [row(w, 32 * ch + p) for w in range(samples) for ch in range(8) for p in range(8)]
    assert len(set(places)) == len(places) >= 4 * k
    for i, p in enumerate(rng.permutation(places)[:k]):
        X[p] = base
        X[p, i % 4] ^= np.uint64((1 << (1 + i % 30)) - 1)
    Q = np.tile(base, (m, 1))
    ri, rd = O.searchbatch("hamming", X, Q[:1], k)
    assert rd.max() <= 30
    idx = ss.GPUExhaustiveSearch(ss.Dist.Bits.Hamming(), ss.MatrixDatabase.from_rows(X), splits=1)
    for _ in range(20):
        ids, dists = ss.searchbatch(idx, ss.GenericContext(), ss.MatrixDatabase.from_rows(Q), k)
        assert np.array_equal(ids.T, np.repeat(ri, m, axis=0))
        assert np.array_equal(dists.T, np.repeat(rd, m, axis=0))


@pytest.mark.parametrize("prec,metric,dim", [("fp32", "sql2", 40), ("fp32", "normcosine", 60), ("bf16", "l2", 96),
                                             ("bf16", "ip", 300), ("fp8", "sql2", 96), ("fp8", "ip", 200)])
@pytest.mark.parametrize("m,k", [(40, 60), (300, 9)])
def test_zero_rows(ss, prec, metric, dim, m, k):
    """Half the rows are zeros, as is every third query."""
    rng = np.random.default_rng(dim + m)
    n = 20_011
    X = rng.standard_normal((n, dim), dtype=np.float32)
    if metric == "normcosine":
        X /= np.linalg.norm(X, axis=1, keepdims=True)
    X[rng.random(n) < 0.5] = 0
    Q = X[rng.integers(0, n, size=m)] + 0.01 * rng.standard_normal((m, dim), dtype=np.float32)
    Q[::3] = 0
    D = {"sql2": ss.Dist.SqL2, "normcosine": ss.Dist.NormCosine, "l2": ss.Dist.L2,
         "ip": ss.Dist.InnerProduct}[metric]()
    got = []
    for s in (0, 1, 17):
        kw = {} if prec == "fp32" else {"precision": prec, "overfetch": 1.25}
        idx = ss.GPUExhaustiveSearch(D, ss.MatrixDatabase.from_rows(X), splits=s, **kw)
        got.append(ss.searchbatch(idx, ss.GenericContext(), ss.MatrixDatabase.from_rows(Q), k))
    for g in got[1:]:
        assert np.array_equal(got[0][0], g[0]) and np.array_equal(got[0][1], g[1])
    ids, dists = got[0]
    if prec == "fp32":
        ri, rd = O.searchbatch(metric, X, Q, k)
        assert np.array_equal(ids.T, ri) and np.array_equal(dists.T, rd)
    elif metric in ("sql2", "l2"):
        zero = np.flatnonzero(~X.any(axis=1))[:k] + 1
        assert np.array_equal(ids.T[::3], np.tile(zero, (len(Q[::3]), 1)))
        assert not dists.T[::3].any()
