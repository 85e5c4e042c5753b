"""Large batches take a first scan (a lane per configuration and robot) before
the warp kernels: verdicts equal the oracle's for every compiled sphere-group
width, fixed and planar bases, joint offsets, box counts around the 32-box
blocks, both types, per-robot masks, step counts given and computed, and inputs
that the FP32 path cannot decide.  The same rows in batches too small for the
scan give the same verdicts, also where a coordinate is not finite or beyond
what a planner samples."""
import numpy as np
import pytest
import torch

from conftest import pkg

pytestmark = pytest.mark.gpu


def _scene(kind):
    scenes = pkg("scenes")
    if kind == "arm50":
        return scenes.make_arm_scene(0, n_boxes=50)
    if kind == "arm22":
        return scenes.make_arm_scene(0, n_boxes=22)
    if kind == "arm8":                                   # eight spheres per link: the widest groups
        return scenes.make_arm_scene(0, n_boxes=32, spheres_per_link=8)
    if kind == "mobile3":
        return scenes.make_mobile_scene(1, n_robots=3, n_boxes=33)
    if kind == "mobile8":
        return scenes.make_mobile_scene(0, n_robots=8, n_boxes=16)
    sc = scenes.make_arm_scene(0, n_boxes=30)
    sc.joint_offset = np.random.default_rng(3).uniform(-1, 1, sc.q_dim)
    return sc


def _inputs(sc, n, dtype, seed):
    scenes = pkg("scenes")
    q = scenes.uniform_configs(sc, n, seed=seed, dtype=np.float64)
    rng = np.random.default_rng(seed)
    for v in (np.nan, np.inf, 3.0e4, -1.0e7, 1.0e10):     # angles and positions past the FP32 path
        q[rng.integers(0, n, 5), rng.integers(0, sc.q_dim, 5)] = v
    return q.astype(dtype)


KINDS = ["arm50", "arm22", "arm8", "mobile3", "mobile8", "offset"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_configurations(gpu, oracle, kind, dtype):
    col = pkg("collision")
    sc = _scene(kind)
    n = 270_001 // len(sc.q_offset)
    q = _inputs(sc, n, dtype, 5)
    s, o = col.Gb300Scene(sc), oracle.OracleScene(sc)
    qd = torch.from_numpy(q).cuda()
    fin = (np.abs(q) < 100).all(1)
    got = s.is_collision_free_batch(qd).cpu().numpy()
    small = torch.cat([s.is_collision_free_batch(c) for c in qd.split(4000)]).cpu().numpy()
    assert np.array_equal(got, small)
    ref = o.configs_free(q[fin])
    assert np.array_equal(got[fin], ref) and 0 < ref.sum() < len(ref)
    mask = 0b101
    got = s.is_collision_free_batch_robots(qd, mask).cpu().numpy()
    small = torch.cat([s.is_collision_free_batch_robots(c, mask) for c in qd.split(4000)]).cpu().numpy()
    assert np.array_equal(got, small)


@pytest.mark.parametrize("kind", ["arm22", "arm8", "mobile3", "offset"])
@pytest.mark.parametrize("dtype,given", [(np.float32, True), (np.float32, False), (np.float64, False)])
def test_edges(gpu, oracle, kind, dtype, given):
    col = pkg("collision")
    sc = _scene(kind)
    n = 270_001 // len(sc.q_offset)
    q1 = _inputs(sc, n, np.float64, 7)
    q1[~np.isfinite(q1) | (np.abs(q1) > 100)] = 0.1
    rng = np.random.default_rng(8)
    q2 = q1 + rng.uniform(-1, 1, q1.shape) * rng.uniform(0.01, 0.8, (n, 1))
    q2[::97] = q1[::97] + 1e-9                            # two steps: no interior position
    q1[:3, 1], q2[:3, 1] = 2.0e5, 2.0e5 + 0.2             # past the FP32 angle reduction
    q1, q2 = q1.astype(dtype), q2.astype(dtype)
    N = rng.integers(2, 40, n).astype(np.int64) if given else None
    s, o = col.Gb300Scene(sc), oracle.OracleScene(sc)
    for kw in (dict(), dict(include_endpoints=True, N_start=1, N_max=7)):
        if given or not kw:
            got = s.is_edge_collision_free_batch(q1, q2, 0.05, N=N, **kw).cpu().numpy()
            assert np.array_equal(got, o.edges_free(q1, q2, 0.05, N=N, **kw)), kw


def test_errors_are_reported(gpu):
    col = pkg("collision")
    sc = _scene("arm22")
    n = 70_000
    q1 = np.zeros((n, sc.q_dim))
    q2 = q1 + 0.1
    s = col.Gb300Scene(sc)
    q2[123, 4] = np.nan
    q2[123, 0] = np.nan
    with pytest.raises(ValueError):
        s.is_edge_collision_free_batch(q1, q2, 0.05)
    q2[123] = 0.1
    with pytest.raises(AssertionError):
        s.is_edge_collision_free_batch(q1, q2, 0.05, N_start=10_000)
