"""More undecided positions than the list has room for: the count stops (at most
one more per warp), the edges whose positions found no place are walked whole,
and listed, lost and ordinary edges side by side equal the oracle."""
import numpy as np
import pytest

from conftest import pkg
from test_gpu_arm import _free_configs, _with_boxes, sparse_arm_scene

pytestmark = pytest.mark.gpu


def _touching(oracle, eps):
    """A scene whose one box lies eps from one sphere of a free configuration, and that configuration."""
    base = sparse_arm_scene(2, n_boxes=0)
    o = oracle.OracleScene(base)
    q = _free_configs(o, base, 1, 11)[0].astype(np.float64)
    c = o.sphere_centers(q)

    def box_at(s, gap):
        lo, hi = c[s] - 0.05, c[s] + 0.05
        lo[0] = c[s][0] + float(base.sphere_radius[s]) + gap
        hi[0] = lo[0] + 0.1
        return _with_boxes(base, lo, hi)

    s = next(s for s in range(len(c)) if oracle.OracleScene(box_at(s, 1e-3)).config_free(q))
    return box_at(s, eps), q


def test_one_long_edge(gpu, oracle):
    scene, q = _touching(oracle, 1e-9)
    steps = 40_000                      # every position undecided; a fresh scene has room for one
    sc = pkg("collision").Gb300Scene(scene)
    N = np.array([steps], dtype=np.int64)
    q1 = q[None]
    q2 = q1.copy()
    got = sc.is_edge_collision_free_batch(q1, q2, 0.05, True, N=N).cpu().numpy()
    assert np.array_equal(got, oracle.OracleScene(scene).edges_free(q1, q2, 0.05, True, N=N))
    assert 1 < sc.last_call_stats()["rechecked_fp64"] <= 1 + 64 * 152


@pytest.mark.parametrize("eps", [-1e-9, 0.0, 1e-9])
@pytest.mark.parametrize("n,steps", [(3, 50), (40, 200)])
def test_listed_and_lost(gpu, oracle, eps, n, steps):
    scene, q = _touching(oracle, eps)
    rng = np.random.default_rng(n)
    q1 = np.tile(q, (n, 1)) + rng.uniform(-1, 1, (n, len(q))) * 1e-7
    q2 = q1 + rng.uniform(-1, 1, (n, len(q))) * 1e-7
    q2[2::3] = q1[2::3] + rng.uniform(-0.3, 0.3, q1[2::3].shape)   # ordinary edges among them
    N = np.full(n, steps, dtype=np.int64)
    o = oracle.OracleScene(scene)
    for incl in (False, True):
        sc = pkg("collision").Gb300Scene(scene)                    # room for n entries
        got = sc.is_edge_collision_free_batch(q1, q2, 0.05, incl, N=N).cpu().numpy()
        assert np.array_equal(got, o.edges_free(q1, q2, 0.05, incl, N=N))
        assert sc.last_call_stats()["rechecked_fp64"] > n          # the list was full
