"""Batches whose lists and minima take more than one pass of the list scan:
the arrays of the XOR + POPC scan, or of smaller calls."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_hamming_in_chunks(ss):
    rng = np.random.default_rng(3)
    X = rng.integers(0, 2**64 - 1, size=(2_000_000, 1), dtype=np.uint64, endpoint=True)
    Q = rng.integers(0, 2**64 - 1, size=(60_001, 1), dtype=np.uint64, endpoint=True)
    idx = ss.GPUExhaustiveSearch(ss.Dist.Bits.Hamming(), ss.MatrixDatabase.from_rows(X))
    ctx = ss.GenericContext()
    a = ss.searchbatch(idx, ctx, ss.MatrixDatabase.from_rows(Q), 5)
    idx.set_param("exact_scan", 1)
    b = ss.searchbatch(idx, ctx, ss.MatrixDatabase.from_rows(Q), 5)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


def test_bf16_in_chunks(ss):
    rng = np.random.default_rng(4)
    X = rng.standard_normal((1_000_000, 32), dtype=np.float32)
    Q = rng.standard_normal((130_003, 32), dtype=np.float32)
    idx = ss.GPUExhaustiveSearch(ss.Dist.SqL2(), ss.MatrixDatabase.from_rows(X), precision="bf16", overfetch=2.0)
    ctx = ss.GenericContext()
    a = ss.searchbatch(idx, ctx, ss.MatrixDatabase.from_rows(Q), 3)
    for s in (slice(0, 50_000), slice(50_000, 100_000), slice(100_000, None)):
        b = ss.searchbatch(idx, ctx, ss.MatrixDatabase.from_rows(Q[s]), 3)
        assert np.array_equal(a[0][:, s], b[0]) and np.array_equal(a[1][:, s], b[1])


def test_device_bytes_count_tiles_and_lists(ss):
    rng = np.random.default_rng(5)
    B = rng.integers(0, 2**64 - 1, size=(50_000, 4), dtype=np.uint64, endpoint=True)
    F = rng.standard_normal((50_000, 64), dtype=np.float32)
    ctx = ss.GenericContext()
    for dist, X, forms in ((ss.Dist.Bits.Hamming(), B, 50_000 * 128), (ss.Dist.SqL2(), F, 50_000 * 3 * 64 * 2)):
        idx = ss.GPUExhaustiveSearch(dist, ss.MatrixDatabase.from_rows(X))
        ss.searchbatch(idx, ctx, ss.MatrixDatabase.from_rows(X[:300]), 10)
        # the rows as given, as FP4 or split BF16 tiles, and 300 x 10 candidates at least
        assert idx.get_param("device_bytes") >= X.nbytes + forms + 300 * 10 * 8
