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


@pytest.mark.parametrize("kind", ["sketches", "fp32", "bf16", "fp8"])
def test_workspace_is_the_calls_own(ss, kind):
    """One query holds no lists for the rows that pad its tile, and calls of
    growing and shrinking sizes find theirs."""
    from oracle import oracle as O
    rng = np.random.default_rng(6)
    ctx = ss.GenericContext()
    if kind == "sketches":
        X = rng.integers(0, 2**64 - 1, size=(20_000, 4), dtype=np.uint64, endpoint=True)
        dist, kw, forms = ss.Dist.Bits.Hamming(), {}, 20_160 * 128
    else:
        X = rng.standard_normal((20_000, 48), dtype=np.float32)
        # operand tiles: at most six bytes an element, padded to 128
        dist, kw, forms = ss.Dist.SqL2(), {} if kind == "fp32" else {"precision": kind, "overfetch": 4.0}, 20_224 * 128 * 6
    idx = ss.GPUExhaustiveSearch(dist, ss.MatrixDatabase.from_rows(X), **kw)
    order = rng.permutation(20_000)
    for call, m in enumerate((1, 3, 40, 1, 300, 7, 700)):
        ids, dists = ss.searchbatch(idx, ctx, ss.MatrixDatabase.from_rows(X[order[:m]]), 5)
        if call == 0:
            assert idx.get_param("device_bytes") < X.nbytes + forms + (1 << 20)
        if kind in ("sketches", "fp32"):
            ri, rd = O.searchbatch("hamming" if kind == "sketches" else "sql2", X, X[order[:m]], 5)
            assert np.array_equal(ids.T, ri) and np.array_equal(dists.T, rd)
        else:
            assert np.array_equal(ids[0], order[:m] + 1)  # each its own nearest


def test_appends_find_their_tiles(ss):
    """Tiles of an index of sketches are allocated for the rows that the
    database has room for: appends within it allocate nothing, and every
    search sees the rows appended before it."""
    from oracle import oracle as O
    rng = np.random.default_rng(8)
    X = rng.integers(0, 2**64 - 1, size=(52_000, 3), dtype=np.uint64, endpoint=True)
    idx = ss.GPUExhaustiveSearch(ss.Dist.Bits.Hamming(), ss.MatrixDatabase.from_rows(X[:30_000]))
    ctx = ss.GenericContext()
    n, held = 30_000, []
    for step in (0, 1, 239, 240, 700, 1, 20_000):
        if step:
            ss.append_items_b(idx, ctx, ss.MatrixDatabase.from_rows(X[n:n + step]))
            n += step
        Q = X[[0, n - 1, n // 2]]
        ids, dists = ss.searchbatch(idx, ctx, ss.MatrixDatabase.from_rows(Q), 4)
        ri, rd = O.searchbatch("hamming", X[:n], Q, 4)
        assert np.array_equal(ids.T, ri) and np.array_equal(dists.T, rd)
        held.append(idx.get_param("device_bytes"))
    # the first append makes room for 45,000 rows, the last one for more
    assert len(set(held[1:6])) == 1
