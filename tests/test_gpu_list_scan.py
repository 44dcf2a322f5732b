"""The list scan (tensor cores, seeded bound, append-only lists) at the edges
of its tiles and lists, and on data that fills its lists: sorted towards the
queries, one tight block that the seed's sample misses, equal rows."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def hamming(ss, X, Q, k, splits=0):
    idx = ss.GPUExhaustiveSearch(ss.Dist.Bits.Hamming(), ss.MatrixDatabase.from_rows(X), splits=splits)
    ids, dists = ss.searchbatch(idx, ss.GenericContext(), ss.MatrixDatabase.from_rows(Q), k)
    ri, rd = O.searchbatch("hamming", X, Q, k)
    assert np.array_equal(ids.T, ri)
    assert np.array_equal(dists.T, rd)


@pytest.mark.parametrize("n,m,words,k,splits", [
    (2048, 32, 16, 1, 0), (20_000, 33, 3, 7, 0), (30_001, 128, 16, 100, 0), (30_207, 129, 5, 10, 3),
    (50_177, 300, 2, 20, 0), (40_000, 257, 1, 10, 1), (70_000, 64, 20, 50, 0), (33_000, 40, 32, 5, 0)])
def test_hamming_shapes(ss, n, m, words, k, splits):
    rng = np.random.default_rng(n + m + words)
    X = rng.integers(0, 2**64 - 1, size=(n, words), dtype=np.uint64, endpoint=True)
    Q = X[rng.integers(0, n, size=m)].copy()
    Q ^= rng.integers(0, 2**64 - 1, size=Q.shape, dtype=np.uint64) & rng.integers(0, 2**64 - 1, size=Q.shape, dtype=np.uint64)
    hamming(ss, X, Q, k, splits)


@pytest.mark.parametrize("kind", ["sorted", "block", "equal"])
@pytest.mark.parametrize("splits", [1, 0])
def test_hamming_full_lists(ss, kind, splits):
    rng = np.random.default_rng(5)
    n, words, k = 24_576, 4, 50
    bits = rng.random((n, words * 64))
    if kind == "sorted":       # every row nearer to the queries than the one before
        X = bits < np.linspace(0.5, 0.02, n)[:, None]
    elif kind == "block":      # 1,700 near rows between two sampled tiles
        X = bits < 0.5
        X[9 * 256:9 * 256 + 1700] = bits[9 * 256:9 * 256 + 1700] < 0.1
    else:
        X = np.repeat(bits[:1] < 0.5, n, axis=0)
    X = np.ascontiguousarray(np.packbits(X, axis=1, bitorder="little")).view(np.uint64)
    Q = np.zeros((40, words), dtype=np.uint64)
    Q[:, 0] = np.arange(40, dtype=np.uint64)
    hamming(ss, X, Q, k, splits)


def clustered(n, dim, rng):
    """Rows sorted towards the query, then a tight block between two sampled tiles."""
    q = rng.standard_normal(dim).astype(np.float32)
    X = rng.standard_normal((n, dim), dtype=np.float32)
    t = np.linspace(0.0, 0.9, n, dtype=np.float32)[:, None]
    X = (1 - t) * X + t * q
    X[9 * 256:9 * 256 + 1700] = q + 0.3 * rng.standard_normal((1700, dim), dtype=np.float32)
    return X, q


@pytest.mark.parametrize("metric,dim", [("sql2", 24), ("cosine", 100), ("normcosine", 64), ("l2", 128), ("ip", 160),
                                        ("cosine", 192)])
@pytest.mark.parametrize("m,k,splits", [(3, 10, 0), (129, 30, 1)])
def test_plain_full_lists(ss, metric, dim, m, k, splits):
    rng = np.random.default_rng(dim + m)
    X, q = clustered(24_600, dim, rng)
    Q = (q + 0.2 * rng.standard_normal((m, dim))).astype(np.float32)
    if metric == "normcosine":
        X /= np.linalg.norm(X, axis=1, keepdims=True)
        Q /= np.linalg.norm(Q, axis=1, keepdims=True)
    dist = {"sql2": ss.Dist.SqL2, "cosine": ss.Dist.Cosine, "normcosine": ss.Dist.NormCosine, "l2": ss.Dist.L2,
            "ip": ss.Dist.InnerProduct}[metric]()
    idx = ss.GPUExhaustiveSearch(dist, ss.MatrixDatabase.from_rows(X), splits=splits)
    ids, dists = ss.searchbatch(idx, ss.GenericContext(), ss.MatrixDatabase.from_rows(Q), k)
    assert idx.get_param("last_plain_tc") == 1.0
    ri, rd = O.searchbatch(metric, X, Q, k)
    assert np.array_equal(ids.T, ri)
    assert np.array_equal(dists.T, rd)


@pytest.mark.parametrize("prec,dim", [("bf16", 96), ("bf16", 300), ("fp8", 130), ("fp8", 768)])
@pytest.mark.parametrize("m,splits", [(1, 0), (200, 1)])
def test_reduced_keys_do_not_depend_on_splits(ss, prec, dim, m, splits):
    """The candidates are the kk smallest approximate keys whatever the splits,
    the sample and the lists' compactions: one split against many."""
    rng = np.random.default_rng(dim)
    X, q = clustered(24_600, dim, rng)
    Q = (q + 0.2 * rng.standard_normal((m, dim))).astype(np.float32)
    got = []
    for s in (splits, 17):
        idx = ss.GPUExhaustiveSearch(ss.Dist.SqL2(), ss.MatrixDatabase.from_rows(X), precision=prec, overfetch=2.0,
                                     splits=s)
        got.append(ss.searchbatch(idx, ss.GenericContext(), ss.MatrixDatabase.from_rows(Q), 20))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])


@pytest.mark.parametrize("metric,dim,k,splits", [("sql2", 24, 10, 0), ("normcosine", 96, 32, 1), ("cosine", 40, 5, 3)])
@pytest.mark.parametrize("n,per", [(66_000, 40), (70_033, 700)])
def test_allknn_locality(ss, metric, dim, k, splits, n, per):
    """allknn in the locality order (clusters smaller and larger than a pivot's
    group, so bounds from the neighbourhood miss or hit) equals the oracle on
    sampled rows and the stored order on all, for the plain method; with
    over-fetched BF16 candidates both orders give the same arrays."""
    rng = np.random.default_rng(n + dim)
    C = rng.standard_normal((n // per, dim), dtype=np.float32)
    X = C[rng.integers(0, C.shape[0], size=n)] + 0.2 * rng.standard_normal((n, dim), dtype=np.float32)
    X[500:540] = X[3]  # equal rows
    if metric == "normcosine":
        X /= np.linalg.norm(X, axis=1, keepdims=True)
    dist = {"sql2": ss.Dist.SqL2, "cosine": ss.Dist.Cosine, "normcosine": ss.Dist.NormCosine}[metric]()
    ctx = ss.GenericContext()
    idx = ss.GPUExhaustiveSearch(dist, ss.MatrixDatabase.from_rows(X), splits=splits)
    ids, dists = ss.allknn(idx, ctx, k)
    rows = np.concatenate([np.arange(490, 545), rng.integers(0, n, size=100)])
    ri, rd = O.searchbatch(metric, X, X[rows], k)
    assert np.array_equal(ids.T[rows], ri) and np.array_equal(dists.T[rows], rd)
    idx.set_param("locality", 0)
    i2, d2 = ss.allknn(idx, ctx, k)
    assert np.array_equal(ids, i2) and np.array_equal(dists, d2)
    idx = ss.GPUExhaustiveSearch(dist, ss.MatrixDatabase.from_rows(X), precision="bf16", overfetch=1.5, splits=splits)
    a = ss.allknn(idx, ctx, k, exclude_self=True)
    idx.set_param("locality", 0)
    b = ss.allknn(idx, ctx, k, exclude_self=True)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


@pytest.mark.parametrize("metric", ["sql2", "l2", "ip", "cosine", "normcosine"])
@pytest.mark.parametrize("prec,dim", [("fp32", 300), ("fp32", 701), ("bf16", 640), ("fp8", 130)])
def test_wide_row_epilogues(ss, metric, prec, dim):
    """Scale, offset or both per row, the query tile resident or streamed: plain
    results are the oracle's; of reduced keys, every row is a candidate of one
    search and what is far behind the k-th of another."""
    rng = np.random.default_rng(dim)
    X, q = clustered(24_600, dim, rng)
    Q = (q + 0.2 * rng.standard_normal((5, dim))).astype(np.float32)
    if metric == "normcosine":
        X /= np.linalg.norm(X, axis=1, keepdims=True)
        Q /= np.linalg.norm(Q, axis=1, keepdims=True)
    dist = {"sql2": ss.Dist.SqL2, "cosine": ss.Dist.Cosine, "normcosine": ss.Dist.NormCosine, "l2": ss.Dist.L2,
            "ip": ss.Dist.InnerProduct}[metric]()
    kw = {} if prec == "fp32" else {"precision": prec, "overfetch": 30.0}
    idx = ss.GPUExhaustiveSearch(dist, ss.MatrixDatabase.from_rows(X), **kw)
    ids, dists = ss.searchbatch(idx, ss.GenericContext(), ss.MatrixDatabase.from_rows(Q), 10)
    ri, rd = O.searchbatch(metric, X, Q, 10)
    if prec == "fp32":
        assert np.array_equal(ids.T, ri)
        assert np.array_equal(dists.T, rd)
    else:
        assert np.mean([len(set(a) & set(b)) for a, b in zip(ids.T, ri)]) >= 9.5
        for j in range(5):  # exact distances of what was found
            pos = {i: d for i, d in zip(ri[j], rd[j])}
            assert all(pos.get(i, d) == d for i, d in zip(ids.T[j], dists.T[j]))
