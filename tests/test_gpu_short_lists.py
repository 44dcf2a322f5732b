"""Few neighbours wanted of many that pass the bound: the finalize's warp shape
with 1 to 3 results and up to a few hundred keys within the bound, and exactly
as many keys as are wanted in its block shape."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

CLOSE = [100, 109, 160, 217, 250, 256, 257]


def sketches(count, place, m, rng):
    """20,000 random sketches of four words, `count` of them within one bit of
    `m` queries that are alike: in one block between sampled tiles, or spread."""
    n, words = 20_000, 4
    X = rng.integers(0, 2**64 - 1, size=(n, words), dtype=np.uint64, endpoint=True)
    base = rng.integers(0, 2**64 - 1, size=words, dtype=np.uint64, endpoint=True)
    at = 9 * 240 + np.arange(count) if place == "block" else np.sort(rng.permutation(n)[:count])
    X[at] = base
    one = rng.random(count) < 0.5
    X[at[one], 0] ^= np.uint64(1) << rng.integers(0, 64, size=one.sum(), dtype=np.uint64)
    Q = np.tile(base, (m, 1))
    Q[:, 1] ^= np.uint64(1) << (np.arange(m, dtype=np.uint64) % np.uint64(64))
    return X, Q


@pytest.mark.parametrize("count", CLOSE)
@pytest.mark.parametrize("place", ["block", "spread"])
@pytest.mark.parametrize("m", [256, 300])
def test_hamming_close_rows(ss, count, place, m):
    rng = np.random.default_rng(count + m)
    X, Q = sketches(count, place, m, rng)
    for splits in (0, 1):
        idx = ss.GPUExhaustiveSearch(ss.Dist.Bits.Hamming(), ss.MatrixDatabase.from_rows(X), splits=splits)
        for k in (1, 2, 3):
            ids, dists = ss.searchbatch(idx, ss.GenericContext(), ss.MatrixDatabase.from_rows(Q), k)
            ri, rd = O.searchbatch("hamming", X, Q, k)
            assert np.array_equal(ids.T, ri)
            assert np.array_equal(dists.T, rd)


@pytest.mark.parametrize("exclude_self,k", [(True, 1), (True, 2), (False, 3)])
def test_hamming_allknn_close_rows(ss, exclude_self, k):
    rng = np.random.default_rng(k)
    X, _ = sketches(230, "block", 1, rng)
    idx = ss.GPUExhaustiveSearch(ss.Dist.Bits.Hamming(), ss.MatrixDatabase.from_rows(X))
    ids, dists = ss.allknn(idx, ss.GenericContext(), k, exclude_self=exclude_self)
    rows = np.concatenate([9 * 240 + np.arange(230), rng.integers(0, X.shape[0], size=60)])
    ri, rd = O.searchbatch("hamming", X, X[rows], k + 1)
    for j, r in enumerate(rows):
        keep = (ri[j] != r + 1) if exclude_self else np.ones(k + 1, bool)
        assert np.array_equal(ids.T[r], ri[j][keep][:k])
        assert np.array_equal(dists.T[r], rd[j][keep][:k])


@pytest.mark.parametrize("prec,dim", [("bf16", 48), ("fp8", 130)])
@pytest.mark.parametrize("overfetch", [1.25, 2.0])
@pytest.mark.parametrize("count", CLOSE)
def test_reduced_close_rows(ss, prec, dim, overfetch, count):
    """Rows stored cluster by cluster, one tight cluster between sampled tiles:
    the candidates do not depend on the splits."""
    rng = np.random.default_rng(count + dim)
    n, m = 24_600, 300
    C = rng.standard_normal((n // 200, dim), dtype=np.float32)
    X = np.repeat(C, 200, axis=0)[:n] + 0.3 * rng.standard_normal((n, dim), dtype=np.float32)
    q = rng.standard_normal(dim).astype(np.float32)
    X[9 * 256:9 * 256 + count] = q + 0.05 * rng.standard_normal((count, dim), dtype=np.float32)
    Q = (q + 0.05 * rng.standard_normal((m, dim))).astype(np.float32)
    got = []
    for s in (0, 1, 17):
        idx = ss.GPUExhaustiveSearch(ss.Dist.SqL2(), ss.MatrixDatabase.from_rows(X), precision=prec,
                                     overfetch=overfetch, splits=s)
        got.append(ss.searchbatch(idx, ss.GenericContext(), ss.MatrixDatabase.from_rows(Q), 1))
    for g in got[1:]:
        assert np.array_equal(got[0][0], g[0]) and np.array_equal(got[0][1], g[1])
    near = ((got[0][0] >= 9 * 256 + 1) & (got[0][0] <= 9 * 256 + count))
    assert near.all()  # of the cluster, whatever the rounding


@pytest.mark.parametrize("exclude_self", [False, True])
@pytest.mark.parametrize("k", [1, 2])
@pytest.mark.parametrize("prec", ["fp32", "bf16"])
def test_locality_close_rows(ss, exclude_self, k, prec):
    rng = np.random.default_rng(7 + k)
    n, dim = 66_000, 40
    C = rng.standard_normal((n // 180, dim), dtype=np.float32)
    X = C[rng.integers(0, C.shape[0], size=n)] + 0.01 * rng.standard_normal((n, dim), dtype=np.float32)
    X[500:740] = X[3]  # equal rows
    kw = {} if prec == "fp32" else {"precision": prec, "overfetch": 1.5}
    idx = ss.GPUExhaustiveSearch(ss.Dist.SqL2(), ss.MatrixDatabase.from_rows(X), **kw)
    a = ss.allknn(idx, ss.GenericContext(), k, exclude_self=exclude_self)
    idx.set_param("locality", 0)
    b = ss.allknn(idx, ss.GenericContext(), k, exclude_self=exclude_self)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    if prec == "fp32" and not exclude_self:
        rows = np.concatenate([np.arange(490, 745), rng.integers(0, n, size=60)])
        ri, rd = O.searchbatch("sql2", X, X[rows], k)
        assert np.array_equal(a[0].T[rows], ri) and np.array_equal(a[1].T[rows], rd)


@pytest.mark.parametrize("k", [1, 5, 40, 150])
@pytest.mark.parametrize("m", [1, 40, 300])
@pytest.mark.parametrize("splits", [0, 1])
def test_exactly_as_many_keys(ss, k, m, splits):
    """The k nearest sketches of every query lie in k groups of the seed's
    sample, so the bound is the k-th distance and exactly k keys are within it."""
    rng = np.random.default_rng(k + m)
    tiles, words = 87, 4
    X = rng.integers(0, 2**64 - 1, size=(tiles * 240, words), dtype=np.uint64, endpoint=True)
    base = rng.integers(0, 2**64 - 1, size=words, dtype=np.uint64, endpoint=True)
    # the sample's tiles and their groups' first rows
    per = 64 if 8 * (tiles // 4) < 4 * k else 8
    samples = max(-(-4 * k // per), tiles // (12 if m <= 256 else 6))
    if 2 * samples >= 4 * k:
        per = 2
    first = {2: [0, 32], 8: range(0, 240, 32), 64: range(0, 240, 4)}[per]
    q = 2 * tiles // 15  # tiles between a unit's 15 atoms of 8 rows

    def row(v, c):  # place c of the sample's v-th unit of 120 rows
        e = v * 15 * q // (2 * samples)
        return (e // 15 + c // 8 * q) * 120 + e % 15 * 8 + c % 8

    places = [row(2 * t + c // 120, c % 120) for t in range(samples) for c in first]
    assert len(places) >= k
    for i, p in enumerate(rng.permutation(places[:k])):
        X[p] = base
        X[p, i % 4] ^= np.uint64((1 << (1 + i % 30)) - 1)  # 1 to 30 bits off; random sketches are 90 and more
    Q = np.tile(base, (m, 1))
    ri, rd = O.searchbatch("hamming", X, Q[:1], k)
    assert rd.max() <= 30
    idx = ss.GPUExhaustiveSearch(ss.Dist.Bits.Hamming(), ss.MatrixDatabase.from_rows(X), splits=splits)
    for _ in range(20):
        ids, dists = ss.searchbatch(idx, ss.GenericContext(), ss.MatrixDatabase.from_rows(Q), k)
        assert np.array_equal(ids.T, np.repeat(ri, m, axis=0))
        assert np.array_equal(dists.T, np.repeat(rd, m, axis=0))
