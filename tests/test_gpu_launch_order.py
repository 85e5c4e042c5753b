"""The kernels of a collision call start before the kernel in front of them has
left the GPU: two batches in alternation on one scene, eagerly and from a
captured graph, give the oracle's verdicts every time (with and without the scan,
none to most of the edges surviving the first position)."""
import numpy as np
import pytest
import torch

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("boxes,n", [(50, 70_000), (50, 3_000), (2, 9_000)])
def test_alternating_batches(gpu, oracle, boxes, n):
    scenes, col, lib = pkg("scenes"), pkg("collision"), pkg("_lib")
    scene = scenes.make_arm_scene(4, n_boxes=boxes)
    sc, o = col.Gb300Scene(scene), oracle.OracleScene(scene)
    rng = np.random.default_rng(n)
    batches = []
    for k in range(2):
        a = scenes.uniform_configs(scene, n, seed=k, dtype=np.float64)
        b = a + rng.uniform(-0.3, 0.3, a.shape)
        N = rng.integers(3, 9, n)
        free = o.configs_free(a)
        edge = o.edges_free(a, b, 0.0, N=N)
        batches.append([torch.from_numpy(x).cuda() for x in (a, b, N)] + [free, edge])
    out = torch.empty(n, dtype=torch.uint8, device="cuda")
    for rep in range(12):
        a, b, N, free, edge = batches[rep % 2]
        assert np.array_equal(sc.is_edge_collision_free_batch(a, b, 0.0, N=N, out=out).cpu().numpy(), edge), rep
        assert np.array_equal(sc.is_collision_free_batch(a, out=out).cpu().numpy(), free), rep
    a, b, N = (x.clone() for x in batches[0][:3])
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    lib.check(sc.lib.mrmg_scene_reserve(sc.h, n, st.cuda_stream))
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        sc.is_edge_collision_free_batch(a, b, 0.0, N=N, out=out, stream=st, flags=lib.MRMG_FLAG_ASYNC)
    for rep in range(12):
        for x, y in zip((a, b, N), batches[rep % 2]):
            x.copy_(y)
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), batches[rep % 2][4]), rep
