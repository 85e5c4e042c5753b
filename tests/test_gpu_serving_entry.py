"""The serving entry points called on their own: mrmg_serving_gather copies
sources of every kind (aligned and not, odd sizes, unused capacity) as numpy
does, and reports tables that do not fit; mrmg_serving_check clears and sets its
error word also for a step without rows."""
import numpy as np
import pytest
import torch

from conftest import pkg

pytestmark = pytest.mark.gpu


def _table(entries, nc, ne):
    """Pinned int64 table: {sources, configurations, edges, 0}, then {address, rows, first row, kind} each."""
    t = torch.zeros(4 + 4 * max(len(entries), 1), dtype=torch.int64).pin_memory()
    t[:3] = torch.tensor([len(entries), nc, ne])
    for i, (a, row, kind) in enumerate(entries):
        t[4 + 4 * i:8 + 4 * i] = torch.tensor([a.data_ptr(), len(a), row, kind])
    return t


def _pinned(a, shift=0):
    """A pinned copy, `shift` elements behind an aligned address."""
    a = torch.from_numpy(np.ascontiguousarray(a))
    flat = torch.empty(a.numel() + shift, dtype=a.dtype).pin_memory()
    out = flat[shift:].view(a.shape)
    out.copy_(a)
    return out


@pytest.mark.parametrize("D", [3, 28])
@pytest.mark.parametrize("shift", [0, 1])
def test_gather(gpu, D, shift):
    lib = pkg("_lib").load()
    rng = np.random.default_rng(D)
    ccap, ecap, sizes = 700, 300, [(513, 1), (1, 200), (100, 40)]
    q1 = torch.full((ccap + ecap, D), -1.0, device="cuda")
    q2, N = q1.clone(), torch.full((ccap + ecap,), -1, dtype=torch.int64, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    w1, w2, wN = q1.cpu().numpy(), q2.cpu().numpy(), np.full(ccap + ecap, 2)
    entries, c0, e0 = [], 0, 0
    for c, e in sizes:
        cfg, a, b = (rng.standard_normal((m, D)).astype(np.float32) for m in (c, e, e))
        n = rng.integers(2, 90, e)
        entries += [(_pinned(cfg, shift), c0, 0), (_pinned(a, shift), e0, 1), (_pinned(b, shift), e0, 2), (_pinned(n), e0, 3)]
        w1[c0:c0 + c] = w2[c0:c0 + c] = cfg
        w1[ccap + e0:ccap + e0 + e], w2[ccap + e0:ccap + e0 + e] = a, b
        wN[c0:c0 + c], wN[ccap + e0:ccap + e0 + e] = 3, n
        c0, e0 = c0 + c, e0 + e
    t = _table(entries, c0, e0)

    def gather(table, cc, ec):
        rc = lib.mrmg_serving_gather(table.data_ptr(), 64, D, cc, ec, q1.data_ptr(), q2.data_ptr(), N.data_ptr(),
                                     err.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        return int(err.cpu())

    assert gather(t, ccap, ecap) == 0
    assert np.array_equal(q1.cpu().numpy(), w1) and np.array_equal(q2.cpu().numpy(), w2)
    assert np.array_equal(N.cpu().numpy(), wN)
    assert gather(_table(entries[:1], c0, ecap + 1), ccap, ecap) != 0      # more edges than there is room for
    err.zero_()
    assert gather(_table([(entries[0][0], 400, 0)], 513, 0), ccap, ecap) != 0   # rows past the capacity
    err.zero_()
    assert gather(_table([], 0, 0), 0, 0) == 0


def test_step_without_rows(gpu):
    lib, col, scenes = pkg("_lib").load(), pkg("collision"), pkg("scenes")
    s = col.Gb300Scene(scenes.make_arm_scene(1, n_boxes=3))
    q = torch.zeros((4, 28), device="cuda")
    N, out = torch.zeros(4, dtype=torch.int64, device="cuda"), torch.zeros(4, dtype=torch.uint8, device="cuda")
    err = torch.full((1,), 7, dtype=torch.int32, device="cuda")
    st, gs = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()

    def check(table):
        rc = lib.mrmg_serving_check(s.h, table.data_ptr(), 8, 0, 0, q.data_ptr(), q.data_ptr(), N.data_ptr(), err.data_ptr(), 0,
                                    out.data_ptr(), st.cuda_stream, gs.cuda_stream)
        torch.cuda.synchronize()
        assert rc == 0
        return int(err.cpu())

    assert check(_table([], 0, 0)) == 0
    assert check(_table([], 1, 0)) != 0
    assert check(_table([], 0, 0)) == 0
