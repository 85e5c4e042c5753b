"""Tensor-core k-NN and radius queries per agent on rows longer than a warp:
agents' slices that leave gaps, reach past coordinate 32 or lie wholly beyond it,
and slices given in another order.  Neighbours, distances and radius sets equal
the oracle's."""
import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,slices", [(40, [[0, 7], [10, 17], [20, 27], [30, 37]]), (33, [[26, 33]]),
                                      (64, [[57, 64], [33, 39], [40, 41]]), (90, [[83, 90], [0, 7], [31, 34]]),
                                      (32, [[25, 32], [0, 2]])])
def test_slices_past_a_warp(gpu, oracle, D, slices):
    knn = pkg("knn")
    rng = np.random.default_rng(D)
    off = np.array([0, 6000, 6050, 7400])
    nodes = rng.uniform(-1, 1, (off[-1], D))
    qs = rng.uniform(-1, 1, (200, D))
    qm = rng.integers(0, 3, 200).astype(np.int32)
    store = knn.NodeStore(nodes, off, slices, "max_euclidean", path="tensor_core")
    for k in (1, 5, 15):
        idx, dist = (t.cpu().numpy() for t in store.knn(qs, qm, k))
        want = oracle.knn(qs, qm, nodes, off, slices, "max_euclidean", k)
        assert np.array_equal(idx, want[0]) and np.array_equal(dist, want[1])
    r = np.asarray(want[1])[:, 9]                       # ten results each
    got = [t.cpu().numpy() for t in store.near(qs, qm, r)]
    for a, b in zip(got, oracle.near(qs, qm, nodes, off, slices, "max_euclidean", r)):
        assert np.array_equal(a, b)
