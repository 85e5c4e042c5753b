"""Near contacts of robots on planar bases and on fixed ones: a box face, and a
sphere of another robot, at a distance that only the exact pass can decide, for
spheres of the base, the first and the last link, one to nine robots."""
import copy

import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu

EPS = [-1e-9, -1e-12, -1e-15, 0.0, 1e-15, 1e-12, 1e-9]


@pytest.mark.parametrize("robots", [1, 3, 9])
def test_planar_box_and_pair_contacts(gpu, oracle, robots):
    scenes, col = pkg("scenes"), pkg("collision")
    base = scenes.make_mobile_scene(robots, n_robots=robots, n_boxes=0)
    # the robots on a wide grid, with joint angles of their own: free
    rng = np.random.default_rng(robots)
    q = rng.uniform(-np.pi, np.pi, base.q_dim)
    for r in range(robots):
        q[9 * r], q[9 * r + 1] = 12.0 * (r % 3), 12.0 * (r // 3)
    o0 = oracle.OracleScene(base)
    assert o0.config_free(q)
    c, rechecked = o0.sphere_centers(q), 0
    rob, rad = np.asarray(base.sphere_robot), np.asarray(base.sphere_radius)
    link = np.asarray(base.sphere_link)
    picks = [rng.choice(np.where((rob == r) & (link == k))[0]) for r in range(robots) for k in (0, 1, 6)]
    for i, s in enumerate(picks):
        k, eps = i % 3, EPS[i % len(EPS)]
        lo, hi = c[s] - 0.01, c[s] + 0.01
        lo[k] = c[s][k] + rad[s] + eps
        hi[k] = lo[k] + 0.01
        scene = copy.deepcopy(base)
        scene.box_lo, scene.box_hi = lo.reshape(1, 3), hi.reshape(1, 3)
        sc, o = col.Gb300Scene(scene), oracle.OracleScene(scene)
        want = o.config_free(q)
        assert sc.is_collision_free_batch(q[None]).item() == want, (s, eps)
        rechecked += sc.last_call_stats()["rechecked_fp64"]
        assert sc.config_free1(q) == bool(want)
        # an edge with the contact at its one interior position
        a, b = q - 0.01, q + 0.01
        assert sc.is_edge_collision_free_batch(a[None], b[None], 0.0, N=np.array([3])).item() \
            == o.edges_free(a[None], b[None], 0.0, N=np.array([3]))[0]
    if robots > 1:   # the last robot moved in x until its lowest sphere and one of robot 0 touch
        sc, o = col.Gb300Scene(base), o0
        for i, eps in enumerate(EPS):
            p = q.copy()
            d0 = 9 * (robots - 1)
            foot0, foot1 = np.where((rob == 0) & (link == 0))[0], np.where((rob == robots - 1) & (link == 0))[0]
            p[d0:d0 + 2] = 0.0
            p[d0 + 1] = q[1] + (c[foot0[0]] - c[foot0].mean(0))[1]
            cc = o.sphere_centers(p)
            gap = np.inf
            for x in foot0:   # the smallest shift along x at which a pair of base spheres touches
                for y in foot1:
                    dy = cc[y][1:] - cc[x][1:]
                    R = rad[x] + rad[y] + eps
                    if (dy ** 2).sum() < R * R:
                        s = cc[x][0] + np.sqrt(R * R - (dy ** 2).sum()) - cc[y][0]
                        gap = s if not np.isfinite(gap) else max(gap, s)
            p[d0] += gap
            assert sc.is_collision_free_batch(p[None]).item() == o.config_free(p), eps
            rechecked += sc.last_call_stats()["rechecked_fp64"]
    assert rechecked > 0
