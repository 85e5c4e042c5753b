"""The FP64 pass of edge checks with one and several undecided positions per
edge: edges that stay at (or move by less than the FP32 band around) a
configuration in contact with a box, so that every checked position is
undecided, and ordinary edges between them.  A batch of one such edge has more
undecided positions than its list has room for (the whole-edge walk)."""
import numpy as np
import pytest

from conftest import pkg
from test_gpu_arm import _free_configs, _with_boxes, sparse_arm_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [-1e-5, -1e-9, 0.0, 1e-9, 1e-5])
@pytest.mark.parametrize("n,steps", [(1, 2), (1, 3), (1, 40), (5, 9), (400, 12)])
def test_undecided_positions(gpu, oracle, eps, n, steps):
    col, scenes = pkg("collision"), pkg("scenes")
    base = sparse_arm_scene(2, n_boxes=0)
    rng = np.random.default_rng(n + steps)
    q = _free_configs(oracle.OracleScene(base), base, 1, 11)[0].astype(np.float64)
    c = oracle.OracleScene(base).sphere_centers(q)

    def box_at(s, gap):
        lo, hi = c[s] - 0.05, c[s] + 0.05
        lo[0] = c[s][0] + float(base.sphere_radius[s]) + gap
        hi[0] = lo[0] + 0.1
        return _with_boxes(base, lo, hi)

    # a sphere whose box touches no other sphere (the box a millimetre away leaves the configuration free)
    alone = [s for s in range(len(c)) if oracle.OracleScene(box_at(s, 1e-3)).config_free(q)]
    scene = box_at(alone[int(rng.integers(len(alone)))], eps)
    q1 = np.tile(q, (n, 1)) + rng.uniform(-1, 1, (n, len(q))) * 1e-7
    q2 = q1 + rng.uniform(-1, 1, (n, len(q))) * 1e-7
    q2[3::4] = q1[3::4] + rng.uniform(-0.3, 0.3, q1[3::4].shape)      # ordinary edges among them
    N = np.full(n, steps, dtype=np.int64)
    sc = col.Gb300Scene(scene)
    o = oracle.OracleScene(scene)
    for incl in (False, True):
        got = sc.is_edge_collision_free_batch(q1, q2, 0.05, incl, N=N).cpu().numpy()
        assert np.array_equal(got, o.edges_free(q1, q2, 0.05, incl, N=N))
        if steps > 2 or incl:
            assert sc.last_call_stats()["rechecked_fp64"] > 0
    # a part of the order, and the same edges through host arrays
    got = sc.is_edge_collision_free_batch(q1, q2, 0.05, True, N=N, N_start=1, N_max=steps - 1).cpu().numpy()
    assert np.array_equal(got, o.edges_free(q1, q2, 0.05, True, N=N, N_start=1, N_max=steps - 1))
    assert np.array_equal(sc.is_edge_collision_free_host(q1, q2, 0.05, True, N=N), o.edges_free(q1, q2, 0.05, True, N=N))
