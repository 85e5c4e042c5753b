"""Distance matrices at the edges of the kernel's forms (coordinates in
registers, staged nodes, nodes read in place; node tiles of 128, query tiles of
16) and of the integer square and root (zeros, subnormals, overflowing squares,
infinities, NaN): bit-identical to the oracle."""
import numpy as np
import pytest

from conftest import pkg

pytestmark = pytest.mark.gpu

METRICS = ["euclidean", "sum_euclidean", "max_euclidean", "max"]


def _same(a, b):
    nan = np.isnan(b)
    return np.array_equal(np.isnan(a), nan) and np.array_equal(a[~nan].view(np.uint64), b[~nan].view(np.uint64))


@pytest.mark.parametrize("Q,M", [(1, 129), (3, 1), (4, 127), (17, 128), (16, 300)])
@pytest.mark.parametrize("per,agents", [(1, 1), (2, 2), (5, 1), (4, 2), (3, 3), (7, 4), (24, 4), (32, 3), (33, 4)])
def test_forms(gpu, oracle, Q, M, per, agents):
    cfg = pkg("configuration")
    rng = np.random.default_rng(Q * 1000 + M + per)
    D = per * agents
    q, x = rng.uniform(-3, 3, (Q, D)), rng.uniform(-3, 3, (M, D))
    x[::5] = q[0]                       # distance 0
    sl = [[i * per, (i + 1) * per] for i in range(agents)]
    for metric in METRICS:
        got = cfg.config_dist_matrix(q, x, sl, metric).cpu().numpy()
        assert _same(got, oracle.dist_matrix(q, x, sl, metric)), metric


@pytest.mark.parametrize("per,agents", [(2, 2), (3, 2), (5, 3)])
def test_value_range(gpu, oracle, per, agents):
    """Coordinates of every size: squares and sums below the normal numbers and
    past the largest one, infinities and NaN among them."""
    cfg = pkg("configuration")
    rng = np.random.default_rng(per)
    D = per * agents
    size = np.exp2(rng.integers(-1070, 1023, (400, D)).astype(np.float64))
    x = rng.uniform(-1, 1, (400, D)) * size
    near = np.exp2(rng.integers(-60, 60, (100, D)).astype(np.float64))
    x[:100] = rng.uniform(-1, 1, (100, D)) * near
    x[100:110, 0], x[110:120, 1], x[120:130, D - 1] = np.inf, np.nan, -np.inf
    x[130:140, 0] = -np.nan
    q = np.concatenate([np.zeros((2, D)), rng.uniform(-1, 1, (4, D)), x[100:103], x[10:20]])
    sl = [[i * per, (i + 1) * per] for i in range(agents)]
    with np.errstate(all="ignore"):
        for metric in METRICS:
            got = cfg.config_dist_matrix(q, x, sl, metric).cpu().numpy()
            assert _same(got, oracle.dist_matrix(q, x, sl, metric)), metric
