"""The integer square and square root of the distance kernels
(csrc/mrmg_exact.cuh), compiled for the host and compared bit for bit with the
host's IEEE instructions.  The FP32 reciprocal root that the square root starts
from is given errors up to 2^-22, more than the device's approximation has."""
import ctypes
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SRC = r"""
#include "mrmg_exact.cuh"
using namespace mrmg;
static uint64_t bits(double d) { uint64_t u; memcpy(&u, &d, 8); return u; }
extern "C" long check_square(const double* x, long n) {
  for (long i = 0; i < n; i++) {
    const uint64_t u = bits(x[i]);
    if (!sq_in_range((uint32_t)(u >> 32))) return -2 - i;
    if (sq_bits((uint32_t)(u >> 32), (uint32_t)u) != bits(x[i] * x[i])) return i;
  }
  return -1;
}
extern "C" long check_sqrt(const double* x, long n, double rel) {
  for (long i = 0; i < n; i++) {
    const uint64_t u = bits(x[i]);
    auto rs = [rel](float f) { return (float)((1.0 + rel) / sqrt((double)f)); };
    if (sqrt_bits((uint32_t)(u >> 32), (uint32_t)u, rs) != bits(sqrt(x[i]))) return i;
  }
  return -1;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("exact")
    (d / "t.cpp").write_text(SRC)
    csrc = ROOT / "multirobot-pathplanning-benchmark_gb300" / "csrc"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I", str(csrc),
                    str(d / "t.cpp"), "-o", str(d / "t.so")], check=True, capture_output=True)
    so = ctypes.CDLL(str(d / "t.so"))
    so.check_square.restype = so.check_sqrt.restype = ctypes.c_long
    so.check_sqrt.argtypes = [ctypes.c_void_p, ctypes.c_long, ctypes.c_double]
    so.check_square.argtypes = [ctypes.c_void_p, ctypes.c_long]
    return so


def _mantissas(rng, n):
    """Random mantissas, and ones at the edges: all zeros, all ones, few bits,
    next to sqrt(2), squares of short numbers and their neighbours."""
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    k = n // 8
    m[:k] = (1 << 52) - 1 - rng.integers(0, 4, k).astype(np.uint64)
    m[k:2 * k] = rng.integers(0, 4, k).astype(np.uint64)
    m[2 * k:3 * k] = np.uint64(1) << rng.integers(0, 52, k).astype(np.uint64)
    m[3 * k:4 * k] = (int(np.float64(np.sqrt(2.0)).view(np.uint64)) & ((1 << 52) - 1)) + \
        rng.integers(-3, 4, k).astype(np.int64).view(np.uint64)
    s = rng.integers(1 << 25, 1 << 26, k).astype(np.float64)
    m[4 * k:5 * k] = ((s * s).view(np.uint64) + rng.integers(-2, 3, k).astype(np.int64).view(np.uint64)) & \
        np.uint64((1 << 52) - 1)
    m[5 * k:6 * k] &= np.uint64(0xffffffff00000000)
    return m


@pytest.mark.parametrize("seed", range(4))
def test_square(lib, seed):
    rng = np.random.default_rng(seed)
    n = 400_000
    e = rng.integers(520, 1521, n).astype(np.uint64)
    e[:2000], e[-2000:] = 520, 1520
    sign = rng.integers(0, 2, n).astype(np.uint64) << np.uint64(63)
    x = np.ascontiguousarray((sign | (rng.permutation(e) << np.uint64(52)) | _mantissas(rng, n)).view(np.float64))
    assert lib.check_square(x.ctypes.data, n) == -1


@pytest.mark.parametrize("rel", [0.0, 2.0 ** -22, -(2.0 ** -22), 2.0 ** -23.5])
def test_square_root(lib, rel):
    rng = np.random.default_rng(11)
    n = 400_000
    e = rng.integers(1, 2047, n).astype(np.uint64)
    e[:2000], e[-2000:] = 1, 2046
    x = np.ascontiguousarray(((rng.permutation(e) << np.uint64(52)) | _mantissas(rng, n)).view(np.float64))
    assert lib.check_sqrt(x.ctypes.data, n, rel) == -1
    # sums of two squares, as the distances give them
    d = rng.uniform(-7, 7, (n, 2))
    x = np.ascontiguousarray(d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1])
    assert lib.check_sqrt(x.ctypes.data, n, rel) == -1
