"""Serving steps that are gathered in parts: part boundaries inside requests,
more sources than a CTA's table, sources on 4-byte addresses, configurations
only and edges only.  Direct steps against packed steps, a sample against the
oracle."""
import ctypes

import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu


def _rows(rng, lim, n, shift):
    buf = np.empty(n * lim.shape[1] + shift, np.float32)
    a = buf[shift:].reshape(n, lim.shape[1])
    a[:] = rng.uniform(lim[0], lim[1], a.shape)
    return a


@pytest.mark.parametrize("sizes", [
    [(140_001, 0)],                         # one source, configurations only
    [(0, 70_003)],                          # edges only
    [(60_000, 999), (3, 45_000), (70_000, 1)],
    [(130, 40)] * 700,                      # 2,800 sources
], ids=["configs", "edges", "uneven", "many"])
@pytest.mark.parametrize("shift", [0, 1])
def test_parts(gpu, oracle, sizes, shift):
    scenes, col, srv, lib = pkg("scenes"), pkg("collision"), pkg("serving"), pkg("_lib")
    v = ctypes.c_int32(0)
    lib.check(lib.load().mrmg_host_access(ctypes.byref(v)))
    if not v.value:
        pytest.skip("the device does not read pageable host memory")
    scene = scenes.make_mobile_scene(0, n_boxes=20)
    lim, rng = np.asarray(scene.limits), np.random.default_rng(len(sizes))
    reqs = [{"configs": _rows(rng, lim, c, shift), "q1": _rows(rng, lim, e, shift), "q2": _rows(rng, lim, e, shift),
             "N": rng.integers(2, 40, e)} for c, e in sizes]
    for r in reqs:   # some edges that are short, so that many of their positions are checked
        r["q2"][::3] = r["q1"][::3] + np.float32(1e-3)
    b = srv.ServingBatcher(col.Gb300Scene(scene), max_sources=4096)
    d, p = b.step(reqs), b.step(reqs, direct=False)
    assert {k[2] for k in b.graphs} == {True, False}
    again = b.step(reqs)
    for x, y, z in zip(d.config_free + d.edge_free, p.config_free + p.edge_free, again.config_free + again.edge_free):
        assert np.array_equal(x, y) and np.array_equal(x, z)
    o = oracle.OracleScene(scene)
    for r, c, e in list(zip(reqs, d.config_free, d.edge_free))[:3]:
        assert np.array_equal(c[-300:], o.configs_free(r["configs"][-300:]))
        assert np.array_equal(e[-100:], o.edges_free(r["q1"][-100:], r["q2"][-100:], 0.0, N=r["N"][-100:]))
