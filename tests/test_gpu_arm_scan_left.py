"""Large batches in which the scan stops because its rows do not collide:
verdicts equal the oracle's for free batches (everything left), for batches that
turn free or begin free (some rows ended, some listed, the rest left), around
the size from which batches are scanned, with two and three rows per warp (sixteen and ten robots),
for edges with and without their endpoints, and for serving steps that are
gathered in parts."""
import copy
import ctypes

import numpy as np
import pytest
import torch

from conftest import pkg

pytestmark = pytest.mark.gpu


def _moved(scene, keep):
    """The scene with all but `keep` boxes carried out of every robot's reach."""
    s = copy.deepcopy(scene)
    s.box_lo[keep:, 0] += 50.0
    s.box_hi[keep:, 0] += 50.0
    return s


def _rows(scene, n, free_at, oracle):
    """n configurations; those with free_at true are free, the others uniform."""
    scenes = pkg("scenes")
    q = scenes.uniform_configs(scene, n, seed=3, dtype=np.float64)
    o = oracle.OracleScene(scene)
    pool = q[o.configs_free(q).astype(bool)]
    m = int(free_at.sum())
    q[free_at] = pool[np.arange(m) % len(pool)] + np.random.default_rng(1).uniform(-1e-4, 1e-4, (m, q.shape[1]))
    return q


N = 80_001
PATTERNS = {"free": np.ones(N, bool), "turns free": np.arange(N) >= 30_000, "begins free": np.arange(N) < 30_000,
            "one in three": np.arange(N) % 3 != 0}


@pytest.mark.parametrize("pattern", list(PATTERNS))
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_patterns(gpu, oracle, pattern, dtype):
    col = pkg("collision")
    scene = pkg("scenes").make_arm_scene(1, n_boxes=17)
    q = _rows(scene, N, PATTERNS[pattern], oracle).astype(dtype)
    s, o = col.Gb300Scene(scene), oracle.OracleScene(scene)
    for n in (65_535, 65_536, N):                          # four robots: scanned from 65,536 rows
        got = s.is_collision_free_batch(torch.from_numpy(q[:n]).cuda()).cpu().numpy()
        assert np.array_equal(got, o.configs_free(q[:n]))
    rng = np.random.default_rng(2)
    q2 = (q + rng.uniform(-1, 1, q.shape) * rng.uniform(0.001, 0.2, (N, 1))).astype(dtype)
    for kw in (dict(), dict(include_endpoints=True, N_start=1, N_max=6)):
        got = s.is_edge_collision_free_batch(q, q2, 0.05, **kw).cpu().numpy()
        assert np.array_equal(got, o.edges_free(q, q2, 0.05, **kw)), kw


@pytest.mark.parametrize("keep", [0, 2, 20])
def test_three_rows_per_warp(gpu, oracle, keep):
    col, scenes = pkg("collision"), pkg("scenes")
    scene = _moved(scenes.make_mobile_scene(1, n_robots=10, n_boxes=20), keep)
    n = 30_000                                             # ten robots: scanned from 26,215 rows
    q = scenes.uniform_configs(scene, n, seed=4, dtype=np.float32)
    # robots apart from one another, so that the rows are free of each other
    side = 3.0 * np.stack(np.meshgrid(np.arange(5), np.arange(2)), -1).reshape(10, 2)
    off = np.asarray(scene.q_offset)
    for r in range(10):
        q[: n // 2, off[r]:off[r] + 2] = side[r] + 0.05 * (q[: n // 2, off[r]:off[r] + 2])
    s, o = col.Gb300Scene(scene), oracle.OracleScene(scene)
    got = s.is_collision_free_batch(torch.from_numpy(q).cuda()).cpu().numpy()
    assert np.array_equal(got, o.configs_free(q))
    q2 = q + np.float32(0.03)
    got = s.is_edge_collision_free_batch(q, q2, 0.01).cpu().numpy()
    assert np.array_equal(got, o.edges_free(q, q2, 0.01))


def test_two_rows_per_warp(gpu, oracle):
    """Sixteen six-joint arms, four groups of four far from one another."""
    col, scenes = pkg("collision"), pkg("scenes")
    one = scenes.make_arm_scene(0, n_boxes=20, n_links=6)
    s = copy.deepcopy(one)
    n = len(one.sphere_radius)
    s.q_offset, s.q_dim = np.arange(16, dtype=np.int32) * 6, 96
    s.base_kind, s.n_links = np.zeros(16, np.int32), np.full(16, 6, np.int32)
    s.base_pose, s.dh = np.tile(one.base_pose, (4, 1)), np.tile(one.dh, (4, 1, 1))
    s.base_pose[:, 9] += 20.0 * (np.arange(16) // 4)
    s.sphere_robot = (np.tile(one.sphere_robot, 4) + 4 * (np.arange(4 * n) // n)).astype(np.int32)
    s.sphere_link, s.sphere_local = np.tile(one.sphere_link, 4), np.tile(one.sphere_local, (4, 1))
    s.sphere_radius, s.limits = np.tile(one.sphere_radius, 4), np.stack([np.full(96, -np.pi), np.full(96, np.pi)])
    for keep in (20, 0):                                   # cluttered for the first group, then free of boxes
        sc = _moved(s, keep)
        q = scenes.uniform_configs(sc, 20_000, seed=4, dtype=np.float32)   # scanned from 16,384 rows
        o = oracle.OracleScene(sc)
        got = col.Gb300Scene(sc).is_collision_free_batch(torch.from_numpy(q).cuda()).cpu().numpy()
        assert np.array_equal(got, o.configs_free(q))
        q2 = q + np.float32(0.1)
        got = col.Gb300Scene(sc).is_edge_collision_free_batch(q, q2, 0.05).cpu().numpy()
        assert np.array_equal(got, o.edges_free(q, q2, 0.05))


@pytest.mark.parametrize("keep", [0, 1])
def test_serving_in_parts(gpu, oracle, keep):
    scenes, col, srv, lib = pkg("scenes"), pkg("collision"), pkg("serving"), pkg("_lib")
    v = ctypes.c_int32(0)
    lib.check(lib.load().mrmg_host_access(ctypes.byref(v)))
    if not v.value:
        pytest.skip("the device does not read pageable host memory")
    scene = _moved(scenes.make_mobile_scene(0, n_boxes=20), keep)
    lim, rng = np.asarray(scene.limits), np.random.default_rng(5)
    grid = 1.9 * np.stack(np.meshgrid(np.arange(4), np.arange(2)), -1).reshape(8, 2)

    def rows(n):
        q = rng.uniform(lim[0], lim[1], (n, lim.shape[1])).astype(np.float32)
        for r in range(8):
            q[: n // 2, 9 * r:9 * r + 2] = grid[r] + 0.05 * q[: n // 2, 9 * r:9 * r + 2]
        return q

    reqs = [{"configs": rows(c), "q1": (a := rows(e)), "q2": a + np.float32(0.01), "N": rng.integers(2, 12, e)}
            for c, e in [(70_000, 20_000), (90_001, 3), (1, 40_000)]]
    b = srv.ServingBatcher(col.Gb300Scene(scene), max_sources=4096)
    d, p, again = b.step(reqs), b.step(reqs, direct=False), b.step(reqs)
    for x, y, z in zip(d.config_free + d.edge_free, p.config_free + p.edge_free, again.config_free + again.edge_free):
        assert np.array_equal(x, y) and np.array_equal(x, z)
    o = oracle.OracleScene(scene)
    for r, c, e in zip(reqs, d.config_free, d.edge_free):
        m, k = min(4000, len(c)), min(2000, len(e))
        assert np.array_equal(c[:m], o.configs_free(r["configs"][:m]))
        assert np.array_equal(e[:k], o.edges_free(r["q1"][:k], r["q2"][:k], 0.0, N=r["N"][:k]))
