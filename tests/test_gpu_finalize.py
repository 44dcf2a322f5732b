"""The selection and re-rank of candidate segments at the edges of its two
shapes (a warp per query up to 256 keys in and 64 out, a block per query
beyond), against the oracle's sequential run: ids and distances identical."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,margin,splits", [(1, 1, 1), (8, 8, 1), (31, 1, 4), (32, 32, 1), (56, 8, 2), (57, 8, 2),
                                             (20, 44, 3), (16, 16, 8), (16, 17, 8), (100, 28, 2), (100, 29, 5)])
@pytest.mark.parametrize("metric,dim", [("sql2", 33), ("cosine", 100), ("normcosine", 64)])
def test_rerank_edges(ss, metric, dim, k, margin, splits):
    rng = np.random.default_rng(100 * k + margin + splits)
    X = rng.standard_normal((5003, dim), dtype=np.float32)
    Q = rng.standard_normal((9, dim), dtype=np.float32)
    if metric == "normcosine":
        X /= np.linalg.norm(X, axis=1, keepdims=True)
        Q /= np.linalg.norm(Q, axis=1, keepdims=True)
    dist = {"sql2": ss.Dist.SqL2, "cosine": ss.Dist.Cosine, "normcosine": ss.Dist.NormCosine}[metric]()
    idx = ss.GPUExhaustiveSearch(dist, ss.MatrixDatabase.from_rows(X), margin=margin, splits=splits)
    ids, dists = ss.searchbatch(idx, ss.GenericContext(), ss.MatrixDatabase.from_rows(Q), k)
    ri, rd = O.searchbatch(metric, X, Q, k)
    assert np.array_equal(ids.T, ri)
    assert np.array_equal(dists.T, rd)


@pytest.mark.parametrize("k,splits", [(64, 4), (65, 4), (64, 5), (1, 7), (600, 8), (5000, 1)])
def test_merge_edges(ss, k, splits):
    rng = np.random.default_rng(k + splits)
    X = rng.standard_normal((5003, 7), dtype=np.float32)
    Q = rng.standard_normal((5, 7), dtype=np.float32)
    idx = ss.GPUExhaustiveSearch(ss.Dist.SqL2(), ss.MatrixDatabase.from_rows(X), exact_scan=1, splits=splits)
    ids, dists = ss.searchbatch(idx, ss.GenericContext(), ss.MatrixDatabase.from_rows(Q), k)
    ri, rd = O.searchbatch("sql2", X, Q, k)
    assert np.array_equal(ids.T, ri)
    assert np.array_equal(dists.T, rd)
    ids, dists = ss.allknn(idx, ss.GenericContext(), min(k, 64), exclude_self=True)
    full, _ = O.searchbatch("sql2", X, X[:200], min(k, 64) + 1)
    want = np.stack([row[row != i + 1][: min(k, 64)] for i, row in enumerate(full)])
    assert np.array_equal(ids.T[:200], want)
