"""Host calls return once every CTA of their launch has reported its results:
calls of one CTA to thousands of CTAs in alternation on one scene, each
compared with the oracle, then calls that take longer than the host polls."""
import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["arm", "discs"])
def test_alternating_sizes(gpu, oracle, kind):
    scenes, col = pkg("scenes"), pkg("collision")
    scene = scenes.make_arm_scene(3, n_boxes=5) if kind == "arm" else scenes.make_disc_scene(0)
    sc, o = col.Gb300Scene(scene), oracle.OracleScene(scene)
    q = (scenes.uniform_configs(scene, 4097, seed=1, dtype=np.float64) if kind == "arm"
         else np.random.default_rng(1).uniform(-2, 2, (4097, 4)))
    a, b = q[:256], q[256:512]
    free, edge = o.configs_free(q), o.edges_free(a, b, 0.05)
    for rep in range(3):
        for n in (1, 4096, 2, 127, 4097, 5, 512):
            assert np.array_equal(sc.is_collision_free_host(q[n % 7:n % 7 + n] if n < 4000 else q[:n]),
                                  free[n % 7:n % 7 + n] if n < 4000 else free[:n]), n
            m = 1 + (n + rep) % 256
            assert np.array_equal(sc.is_edge_collision_free_host(a[:m], b[:m], 0.05), edge[:m]), m
    # every position of 200 fine edges
    fine = 2e-3
    assert np.array_equal(sc.is_edge_collision_free_host(a[:200], b[:200], fine), o.edges_free(a[:200], b[:200], fine))
    assert sc.is_collision_free_host(q[:1])[0] == free[0]
