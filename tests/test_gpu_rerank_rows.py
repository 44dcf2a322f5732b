"""Row kernels at the edges of their staging (32 dimensions at a time, 16-byte
copies or not): rerank! and the row norms against the oracle's sequential run,
ids and distances identical, and the network's products at every tile width
against FP64."""
import numpy as np
import pytest

from oracle import mlp_oracle as MO
from oracle import oracle as O
from test_gpu_learned import gpu_grads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [1, 2, 127, 128, 129, 300])
@pytest.mark.parametrize("metric,dim", [("sql2", 1), ("l2", 33), ("cosine", 96), ("normcosine", 130), ("ip", 64),
                                        ("hamming", 3)])
def test_rerank_lengths(ss, metric, dim, length):
    rng = np.random.default_rng(1000 * length + dim)
    if metric == "hamming":
        X = rng.integers(0, 2**63, size=(500, dim), dtype=np.uint64)
        Q = rng.integers(0, 2**63, size=(7, dim), dtype=np.uint64)
    else:
        X = rng.standard_normal((500, dim), dtype=np.float32)
        Q = rng.standard_normal((7, dim), dtype=np.float32)
        if metric == "normcosine":
            X /= np.linalg.norm(X, axis=1, keepdims=True)
            Q /= np.linalg.norm(Q, axis=1, keepdims=True)
    dist = {"sql2": ss.Dist.SqL2, "l2": ss.Dist.L2, "cosine": ss.Dist.Cosine, "normcosine": ss.Dist.NormCosine,
            "ip": ss.Dist.InnerProduct, "hamming": ss.Dist.Bits.Hamming}[metric]()
    idx = ss.GPUExhaustiveSearch(dist, ss.MatrixDatabase.from_rows(X))
    cand = np.stack([rng.permutation(500)[:length] + 1 for _ in range(7)], axis=1).astype(np.uint32)
    cand[length // 2:, 1::3] = 0  # some lists end early, one at once where they are of one id
    ids = np.asfortranarray(cand.copy())
    dists = np.asfortranarray(np.full((length, 7), 7.0, np.float32))
    ss.rerank_b(idx, ss.MatrixDatabase.from_rows(Q), ids, dists)
    for j in range(7):
        ri, rd = O.rerank(metric, X, Q[j], cand[:, j], np.full(length, 7.0, np.float32))
        assert np.array_equal(ids[:, j], ri)
        assert np.array_equal(dists[ri != 0, j], rd[ri != 0])
        assert np.all(dists[ri == 0, j] == 7.0)  # what is behind a list's end stays


@pytest.mark.parametrize("d,H,E,B", [(48, 100, 40, 400), (48, 256, 30, 1700), (70, 250, 64, 3400)])
def test_product_tile_widths(ss, d, H, E, B):
    """32, 64 and 128 columns per tile of the hidden gradient (and of what
    else has few tiles); the tolerance is the gradient check's own: FP32
    accumulation, 1e-4 of the largest entry."""
    rng = np.random.default_rng(d + H + E)
    W1 = (rng.standard_normal((H, d)) * np.sqrt(2.0 / d)).astype(np.float32)
    b1 = (rng.standard_normal(H) * 0.1).astype(np.float32)
    W2 = (rng.standard_normal((E, H)) * np.sqrt(1.0 / H)).astype(np.float32)
    b2 = (rng.standard_normal(E) * 0.1).astype(np.float32)
    X = rng.standard_normal((3 * B, d)).astype(np.float32)
    X[B:] = np.concatenate([X[:B], X[:B]]) + 0.5 * X[B:]
    _, _, z = MO.forward(W1, b1, W2, b2, X)
    gap = np.sort(((z[:B] - z[2 * B:]) ** 2).sum(1) - ((z[:B] - z[B:2 * B]) ** 2).sum(1))
    mid = B // 2 - 20 + int(np.argmax(np.diff(gap[B // 2 - 20:B // 2 + 20])))  # the widest gap near the median
    margin = float(0.5 * (gap[mid] + gap[mid + 1]))
    loss, *grads = gpu_grads(ss, W1, b1, W2, b2, X, margin)
    rl, *want = MO.triplet_loss_and_grads(W1, b1, W2, b2, X, margin)
    assert abs(loss - rl) <= 1e-4 * max(1.0, abs(rl))
    for i, (g, r) in enumerate(zip(grads, want)):
        scale = max(np.abs(r).max(), np.abs(want[2]).max() if i == 3 else 0.0)
        assert np.abs(g - r).max() <= 1e-4 * scale


@pytest.mark.parametrize("rows,dim", [(1, 1), (31, 3), (32, 31), (33, 32), (64, 33), (65, 64), (200, 130)])
def test_row_norms(ss, rows, dim):
    """Cosine divides by the norms of both sides: a norm off in its last bit shows."""
    rng = np.random.default_rng(rows + dim)
    X = rng.standard_normal((rows, dim), dtype=np.float32)
    Q = rng.standard_normal((rows, dim), dtype=np.float32)
    k = min(rows, 5)
    idx = ss.GPUExhaustiveSearch(ss.Dist.Cosine(), ss.MatrixDatabase.from_rows(X), exact_scan=1)
    ids, dists = ss.searchbatch(idx, ss.GenericContext(), ss.MatrixDatabase.from_rows(Q), k)
    ri, rd = O.searchbatch("cosine", X, Q, k)
    assert np.array_equal(ids.T, ri)
    assert np.array_equal(dists.T, rd)


@pytest.mark.parametrize("m,k,splits", [(3, 10, 300), (3, 10, 256), (200, 60, 257)])
def test_many_lists(ss, m, k, splits):
    """More than 512 candidate lists per query are walked, fewer gathered flat."""
    rng = np.random.default_rng(m + splits)
    X = rng.standard_normal((80_000, 8), dtype=np.float32)
    Q = rng.standard_normal((m, 8), dtype=np.float32)
    idx = ss.GPUExhaustiveSearch(ss.Dist.SqL2(), ss.MatrixDatabase.from_rows(X), splits=splits)
    ids, dists = ss.searchbatch(idx, ss.GenericContext(), ss.MatrixDatabase.from_rows(Q), k)
    ri, rd = O.searchbatch("sql2", X, Q, k)
    assert np.array_equal(ids.T, ri)
    assert np.array_equal(dists.T, rd)
