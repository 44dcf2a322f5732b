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
