"""Penetration kernels at the edges of their packing: odd sphere counts per
robot (padded with an empty sphere), 0 to 5 boxes (pairs of boxes, a pair per
half warp), path lengths around 16 and 32 waypoints, few segments (clusters of
CTAs) and many, and a beta on each side of the bound of the direct form.  The
reference is the float64 autograd restatement, with the tolerances of
test_gpu_penetration.py (cost 1e-5, gradient 1e-4)."""
import dataclasses

import numpy as np
import pytest
import torch

from conftest import pkg

pytestmark = pytest.mark.gpu

COST_RTOL = 1e-5
GRAD_RTOL = 1e-4


def _scene(n_boxes, drop):
    """The four-arm scene without the spheres of index % drop == 0."""
    sc = pkg("scenes").make_arm_scene(0, n_boxes=max(n_boxes, 1))
    keep = np.arange(len(sc.sphere_radius)) % drop != 0 if drop else np.ones(len(sc.sphere_radius), bool)
    return dataclasses.replace(
        sc, sphere_robot=sc.sphere_robot[keep], sphere_link=sc.sphere_link[keep], sphere_local=sc.sphere_local[keep],
        sphere_radius=sc.sphere_radius[keep], box_lo=sc.box_lo[:n_boxes], box_hi=sc.box_hi[:n_boxes])


@pytest.mark.parametrize("n_boxes,drop,T,P", [(0, 5, 15, 1), (1, 0, 16, 2), (2, 5, 17, 1), (3, 9, 33, 2), (5, 41, 1, 3),
                                              (4, 2, 47, 1), (3, 5, 20, 200)])
@pytest.mark.parametrize("beta", [1.0, 60.0])
def test_cost_and_gradient(gpu, n_boxes, drop, T, P, beta):
    import penetration_f64 as orc_pen

    pen, col, scenes = pkg("penetration"), pkg("collision"), pkg("scenes")
    sc = _scene(n_boxes, drop)
    paths = scenes.make_path_workload(sc, seed=3 + T, n_paths=P, n_waypoints=T)
    s = col.Gb300Scene(sc)
    assert pen.penetration_info(s)["spheres"] == len(sc.sphere_radius)
    prm = pen.PenetrationParams(beta=beta)
    w = torch.from_numpy(paths).cuda()
    both = pen.path_penetration(s, w, prm, cost=True, waypoint_cost=True, grad=True)
    cost = pen.path_penetration(s, w, prm)["cost"].cpu().numpy()
    grad = pen.path_penetration(s, w, prm, cost=False, grad=True)["grad"]
    assert torch.equal(grad, both["grad"])
    n = min(P, 3)
    c_ref, g_ref = orc_pen.penetration_grad(sc.arrays(), paths[:n], beta=beta)
    for c in (cost[:n], both["cost"].cpu().numpy()[:n], both["waypoint_cost"].double().sum(1).cpu().numpy()[:n]):
        assert np.all(np.abs(c - c_ref) <= COST_RTOL * np.abs(c_ref))
    g = grad.cpu().numpy().astype(np.float64)
    for p in range(n):
        assert np.linalg.norm(g[p] - g_ref[p]) <= GRAD_RTOL * np.linalg.norm(g_ref[p])
