"""A path's penetration cost, per-waypoint cost and gradient have the same bits
alone and in any batch: few segments are shared by clusters of 2, 4 or 8 CTAs,
many are not, and the sums are the same.  Both segment lengths, tasks of one and
of many turns per warp, and the gradient in groups of robots."""
import pytest
import torch

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,T,warps", [("arm", 45, 0), ("arm", 17, 4), ("arm", 33, 7), ("few", 100, 0), ("two", 20, 2),
                                          ("mobile8", 40, 0)])
def test_bits_do_not_depend_on_the_batch(gpu, kind, T, warps):
    pen, col, scenes = pkg("penetration"), pkg("collision"), pkg("scenes")
    sc = {"arm": lambda: scenes.make_arm_scene(0, n_boxes=21),
          "few": lambda: scenes.make_arm_scene(1, n_boxes=3),
          "two": lambda: scenes.make_mobile_scene(1, n_robots=2, n_boxes=30),
          "mobile8": lambda: scenes.make_mobile_scene(0)}[kind]()
    s = col.Gb300Scene(sc)
    w = torch.from_numpy(scenes.make_path_workload(sc, seed=T, n_paths=700, n_waypoints=T)).cuda()

    def run(x):
        kw = dict(warps_per_cta=warps)
        return [*pen.path_penetration(s, x, waypoint_cost=True, grad=True, **kw).values(),
                *pen.path_penetration(s, x, waypoint_cost=True, **kw).values(),
                *pen.path_penetration(s, x, cost=False, grad=True, **kw).values()]

    whole = run(w)
    for n in (1, 2, 7, 13, 40, 90):
        for a, b in zip(run(w[:n].contiguous()), whole):
            assert torch.equal(a, b[:n]), n
