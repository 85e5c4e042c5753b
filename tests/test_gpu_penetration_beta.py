"""Very small and very large beta: the places without a sphere or a box (odd
sphere counts, odd box counts) add nothing, whatever scales them.  The
reference is the float64 autograd restatement, with the tolerances of
test_gpu_penetration.py (cost 1e-5, gradient 1e-4)."""
import numpy as np
import pytest
import torch

from conftest import pkg
from test_gpu_penetration_forms import COST_RTOL, GRAD_RTOL, _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_boxes,drop,T,P", [(3, 5, 17, 2), (0, 9, 33, 1), (5, 5, 20, 200)])
@pytest.mark.parametrize("beta", [1e-30, 1e-28, 1e-20, 1e32])
def test_extreme_beta(gpu, oracle, n_boxes, drop, T, P, beta):
    import penetration_f64 as orc_pen

    pen, col, scenes = pkg("penetration"), pkg("collision"), pkg("scenes")
    sc = _scene(n_boxes, drop)
    assert any(np.bincount(sc.sphere_robot) % 2)
    paths = scenes.make_path_workload(sc, seed=3 + T, n_paths=P, n_waypoints=T)
    s = col.Gb300Scene(sc)
    w = torch.from_numpy(paths).cuda()
    both = pen.path_penetration(s, w, pen.PenetrationParams(beta=beta), cost=True, grad=True)
    cost = pen.path_penetration(s, w, pen.PenetrationParams(beta=beta))["cost"].cpu().numpy()
    n = min(P, 2)
    c_ref, g_ref = orc_pen.penetration_grad(sc.arrays(), paths[:n], beta=beta)
    for c in (cost[:n], both["cost"].cpu().numpy()[:n]):
        assert np.all(np.abs(c - c_ref) <= COST_RTOL * np.abs(c_ref))
    if beta < 1:                       # (a huge beta's gradient is a step, decided by the last bit of a distance)
        g = both["grad"].cpu().numpy().astype(np.float64)
        for p in range(n):
            assert np.linalg.norm(g[p] - g_ref[p]) <= GRAD_RTOL * np.linalg.norm(g_ref[p])
