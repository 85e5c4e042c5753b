"""Radius queries at the edges of their forms: result counts around the 48 that
are staged per query, rows that are loaded whole and rows that are not (27 and
9 coordinates, agents that leave a gap), modes shorter than a bitmap word, both
query paths.  Index sets and distances equal the oracle's."""
import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("path", ["tensor_core", "exact"])
@pytest.mark.parametrize("metric", ["euclidean", "max_euclidean"])
@pytest.mark.parametrize("slices", [[[0, 7], [7, 14], [14, 21], [21, 28]], [[0, 7], [7, 14], [14, 21], [21, 27]],
                                    [[0, 4], [4, 9]], [[0, 3], [4, 8]]])
def test_result_counts(gpu, oracle, path, metric, slices):
    knn = pkg("knn")
    D = slices[-1][1]
    rng = np.random.default_rng(D)
    sizes = [5000, 31, 1, 0, 700]
    off = np.concatenate([[0], np.cumsum(sizes)])
    nodes = rng.uniform(-1, 1, (off[-1], D))
    qs = rng.uniform(-1, 1, (150, D))
    qm = rng.choice([0, 1, 2, 3, 4], 150, p=[0.6, 0.1, 0.1, 0.1, 0.1]).astype(np.int32)
    r = np.zeros(150)
    for i, q in enumerate(qs):
        x = nodes[off[qm[i]]:off[qm[i] + 1]]
        if len(x) == 0:
            r[i] = 1.0
            continue
        d = q - x
        if metric == "euclidean":
            dist = np.sqrt((d[:, :slices[-1][1]] ** 2).sum(1))
        else:
            dist = np.max([np.sqrt((d[:, s:e] ** 2).sum(1)) for s, e in slices], axis=0)
        k = min([0, 1, 46, 47, 48, 200, 3000][i % 7], len(x) - 1)
        r[i] = np.sort(dist)[k]          # k + 1 results: 1, 2, 47, 48, 49, 201, 3001
    store = knn.NodeStore(nodes, off, slices, metric, path=path)
    offs, idx, dist = (t.cpu().numpy() for t in store.near(qs, qm, r))
    want = oracle.near(qs, qm, nodes, off, slices, metric, r)
    for a, b in zip((offs, idx, dist), want):
        assert np.array_equal(a, b)
    # a capacity below the total: fetched afterwards
    offs, idx, dist = (t.cpu().numpy() for t in store.near(qs, qm, r, cap=100))
    assert np.array_equal(idx, want[1]) and np.array_equal(dist, want[2])
