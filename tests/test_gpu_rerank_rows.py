"""The FP64 re-rank of neighbours reads whole rows where their layout allows it:
aligned and unaligned queries, rows of whole 32-byte words and others, few and
many (equal) candidates, coordinates that are infinite or NaN."""
import numpy as np
import pytest
import torch

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("path", ["tensor_core", "auto"])
@pytest.mark.parametrize("metric", ["euclidean", "max_euclidean"])
@pytest.mark.parametrize("slices", [[[0, 7], [7, 14], [14, 21], [21, 28]], [[0, 3], [3, 8]], [[0, 4], [4, 9]]])
def test_rows(gpu, oracle, path, metric, slices):
    knn = pkg("knn")
    D, k = slices[-1][1], 10
    rng = np.random.default_rng(D)
    nodes = rng.uniform(-1, 1, (6000, D))
    nodes[1000:1040] = nodes[1000]           # 40 equal rows: more candidates than lanes
    off = np.array([0, 4000, 4005, 6000])
    Q = 3 if path == "auto" else 140
    qs = rng.uniform(-1, 1, (Q, D))
    qs[0] = nodes[1000] + 1e-3
    qm = rng.integers(0, 3, Q).astype(np.int32)
    qm[0] = 0
    store = knn.NodeStore(nodes, off, slices, metric, path=path)
    buf = torch.empty(Q * D + 1, dtype=torch.float64, device="cuda")
    got = []
    for shift in (0, 1):
        v = buf[shift:shift + Q * D].view(Q, D)
        v.copy_(torch.from_numpy(qs))
        got.append([t.cpu().numpy() for t in (*store.knn(v, qm, k), *store.near(v, qm, 0.6))])
    want = [*oracle.knn(qs, qm, nodes, off, slices, metric, k),
            *oracle.near(qs, qm, nodes, off, slices, metric, np.full(Q, 0.6))]
    for g in got:
        for a, b in zip(g, want):
            assert np.array_equal(a, b)
    # a coordinate that is no number (first agent, last agent): the layout does not matter
    bad = [np.nan, np.inf, -np.inf]
    for j, c in ((0, 0), (1, D - 1), (2, D - 1)):
        qs[j, c] = bad[j]
    got = []
    for shift in (0, 1):
        v = buf[shift:shift + Q * D].view(Q, D)
        v.copy_(torch.from_numpy(qs))
        got.append([t.cpu().numpy() for t in (*store.knn(v, qm, k), *store.near(v, qm, 0.6))])
    for a, b in zip(*got):
        assert np.array_equal(a, b)
