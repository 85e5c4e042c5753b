"""The count of undecided edge positions (csrc/mrmg_pending.cuh), compiled for
the host: near the end of an int, with scratch blocks below, at and above it,
it neither wraps nor hands out a place past the list, also when no warp ever sees
another one's note that the list is full."""
import ctypes
import subprocess

import pytest

from conftest import ROOT

SRC = r"""
#include "mrmg_pending.cuh"
using namespace mrmg;
struct Warp {
  int* count;
  bool full = false;                  // only its own note
  bool lost() const { return full; }
  int add() { return (*count)++; }
  void lose() { full = true; }
};
// `warps` warps find `each` positions, starting from `start` listed ones; out:
// final count, places given out, lowest and highest place, entries to read
extern "C" void run(long long cap, int start, int warps, int each, long long* out) {
  Warp* w = new Warp[warps];
  int count = start;
  long long given = 0, lo = 1ll << 40, hi = -1;
  for (int i = 0; i < warps; i++) w[i].count = &count;
  for (int k = 0; k < each; k++)
    for (int i = 0; i < warps; i++) {
      const int s = pend_claim(w[i], cap);
      if (s == -1) continue;
      given++;
      lo = s < lo ? s : lo;
      hi = s > hi ? s : hi;
    }
  out[0] = count; out[1] = given; out[2] = lo; out[3] = hi; out[4] = pend_listed(count, cap);
  delete[] w;
}
"""
MAX = 2 ** 31 - 2 ** 26


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("pending")
    (d / "t.cpp").write_text(SRC)
    csrc = ROOT / "multirobot-pathplanning-benchmark_gb300" / "csrc"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fwrapv", "-shared", "-fPIC", "-I", str(csrc), str(d / "t.cpp"), "-o",
                    str(d / "t.so")], check=True, capture_output=True)
    so = ctypes.CDLL(str(d / "t.so"))
    so.run.argtypes = [ctypes.c_longlong, ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
    return so


@pytest.mark.parametrize("cap,start", [(1, 0), (1, 1), (1000, 990), (MAX - 1, MAX - 7), (MAX, MAX - 3), (MAX, MAX),
                                       (2 ** 31 - 1, MAX - 5), (2 ** 32, MAX - 5), (2 ** 33, 0)])
def test_count_stops_at_the_list(lib, cap, start):
    warps, each = 9728, 300            # 64 warps on each of 152 SMs; 2.9 M positions
    out = (ctypes.c_longlong * 5)()
    lib.run(cap, start, warps, each, out)
    count, given, lo, hi, listed = out
    room = min(cap, MAX)
    assert given == min(room - start, warps * each) and (given == 0 or (lo, hi) == (start, start + given - 1))
    assert 0 < count <= room + warps < 2 ** 31
    assert listed == start + given
