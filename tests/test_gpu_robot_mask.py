"""Checks of some of the robots on scenes whose lanes own several sphere groups:
a robot outside the mask does not count, also where a box touches both it and a
robot inside whose groups share its lanes.  Large batches (with the scan), small
ones and single calls equal the oracle."""
import numpy as np
import pytest
import torch

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_robots,n_boxes,mask", [(8, 16, 0b101), (8, 60, 0b10010), (8, 9, 0b11110000), (8, 200, 1 << 7),
                                                   (3, 33, 0b010), (5, 20, 0b10001)])
def test_masks(gpu, oracle, n_robots, n_boxes, mask):
    col, scenes = pkg("collision"), pkg("scenes")
    sc = scenes.make_mobile_scene(0, n_robots=n_robots, n_boxes=n_boxes)
    n = 270_001 // n_robots
    q = scenes.uniform_configs(sc, n, seed=5, dtype=np.float64)
    want = oracle.OracleScene(sc).configs_free_for_robots(q, mask)
    s, qd = col.Gb300Scene(sc), torch.from_numpy(q).cuda()
    got = s.is_collision_free_batch_robots(qd, mask).cpu().numpy()
    assert np.array_equal(got, want)
    for m in (4000, 1000):
        small = torch.cat([s.is_collision_free_batch_robots(c, mask) for c in qd[:12_000].split(m)]).cpu().numpy()
        assert np.array_equal(small, want[:12_000])
