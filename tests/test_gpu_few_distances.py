"""Distances in FP64 instructions and in integer squares and roots, on both sides
of each rule that chooses: matrices of nodes read in place around 2^18
distances, exact k-NN around two warps per scheduler and with lists past 16,
radius queries around the same and with chunks of several words per warp.
Everything equals the oracle bit for bit."""
import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu

FOUR = [[0, 7], [7, 14], [14, 21], [21, 28]]


@pytest.mark.parametrize("D", [97, 128, 129])
@pytest.mark.parametrize("Q,M", [(1, 300), (6, 43_690), (6, 43_691), (17, 20_000)])
def test_matrix_in_place(gpu, oracle, D, Q, M):
    cfg = pkg("configuration")
    rng = np.random.default_rng(D + Q)
    q, x = rng.uniform(-1, 1, (Q, D)), rng.uniform(-1, 1, (M, D))
    x[:3], x[3, 5], x[4, 7] = q[0], np.nan, np.inf
    sl = [[0, D // 2], [D // 2, D]]
    for metric in ("euclidean", "sum_euclidean", "max_euclidean", "max"):
        got = cfg.config_dist_matrix(q, x, sl, metric).cpu().numpy()
        assert np.array_equal(got, oracle.dist_matrix(q, x, sl, metric), equal_nan=True), metric


@pytest.mark.parametrize("metric", ["sum_euclidean", "max_euclidean", "max"])
@pytest.mark.parametrize("Q", [1, 10, 11, 60])
def test_knn_around_the_rule(gpu, oracle, metric, Q):
    knn = pkg("knn")
    rng = np.random.default_rng(Q)
    off = np.array([0, 30_000, 30_300])                 # 118 chunks: 1,180 warps for ten queries, 1,298 for eleven
    nodes = rng.uniform(-1, 1, (off[-1], 28))
    nodes[7] = nodes[9]
    qs = rng.uniform(-1, 1, (Q, 28))
    qs[0] = nodes[9]
    qm = np.zeros(Q, dtype=np.int32)
    store = knn.NodeStore(nodes, off, FOUR, metric, path="exact")
    for k in (1, 15, 16, 17, 40):
        idx, dist = (t.cpu().numpy() for t in store.knn(qs, qm, k))
        want = oracle.knn(qs, qm, nodes, off, FOUR, metric, k)
        assert np.array_equal(idx, want[0]) and np.array_equal(dist, want[1]), k


@pytest.mark.parametrize("Q", [40, 1216, 1217, 2100])
def test_knn_warp_per_query(gpu, oracle, Q):
    knn = pkg("knn")
    rng = np.random.default_rng(Q)
    off = np.array([0, 400, 777])
    nodes, qs = rng.uniform(-1, 1, (off[-1], 6)), rng.uniform(-1, 1, (Q, 6))
    qm = rng.integers(0, 2, Q).astype(np.int32)
    sl = [[0, 3], [3, 6]]
    for k in (3, 20):
        idx, dist = (t.cpu().numpy() for t in knn.knn_exact(qs, qm, nodes, off, sl, "sum_euclidean", k))
        want = oracle.knn(qs, qm, nodes, off, sl, "sum_euclidean", k)
        assert np.array_equal(idx, want[0]) and np.array_equal(dist, want[1]), k


@pytest.mark.parametrize("metric,Q", [("sum_euclidean", 1), ("sum_euclidean", 2), ("max", 3), ("euclidean", 2),
                                      ("max_euclidean", 9)])
def test_near_exact_path(gpu, oracle, metric, Q):
    knn = pkg("knn")
    rng = np.random.default_rng(Q)
    off = np.array([0, 30_000])                         # 938 words a query
    for D, sl in ((28, FOUR), (27, [[0, 9], [9, 18], [18, 27]])):
        nodes, qs = rng.uniform(-1, 1, (off[-1], D)), rng.uniform(-1, 1, (Q, D))
        qm = np.zeros(Q, dtype=np.int32)
        r = np.asarray(oracle.knn(qs, qm, nodes, off, sl, metric, 60)[1])[:, -1]
        got = [t.cpu().numpy() for t in knn.NodeStore(nodes, off, sl, metric, path="exact").near(qs, qm, r)]
        for a, b in zip(got, oracle.near(qs, qm, nodes, off, sl, metric, r)):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("D,sl", [(4, [[0, 2], [2, 4]]), (6, [[0, 3], [3, 6]])])
def test_near_in_chunks_of_words(gpu, oracle, D, sl):
    knn = pkg("knn")
    rng = np.random.default_rng(D)
    off = np.array([0, 14_001, 14_001, 40_001, 40_021])  # 2.1 M words in all: two or more turns per chunk
    nodes, qs = rng.uniform(-1, 1, (off[-1], D)), rng.uniform(-1, 1, (4096, D))
    qm = rng.choice([0, 1, 2, 3], 4096, p=[0.45, 0.05, 0.4, 0.1]).astype(np.int32)
    r = np.where(rng.uniform(size=4096) < 0.02, 0.5, 0.12)  # a few queries with hundreds of results
    r[qm == 3] = 0.9
    got = [t.cpu().numpy() for t in knn.NodeStore(nodes, off, sl, "euclidean", path="tensor_core").near(qs, qm, r)]
    for a, b in zip(got, oracle.near(qs, qm, nodes, off, sl, "euclidean", r)):
        assert np.array_equal(a, b)
