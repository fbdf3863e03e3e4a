"""The tuner's rule for the hand-off threshold (csrc/hh_handoff.h), compiled for the host and
given made-up launch times: differences of a percent, the noise of a timing, leave the default;
a threshold that is clearly faster is found from there; an error ends the choice."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = """
#include "hh_handoff.h"
typedef int (*run_t)(int, int, float *);
extern "C" int pick(int def, run_t run, int *div, int *mul) {
  return hh::pick_handoff(def, [&](int d, int m, float *ms) { return run(d, m, ms); }, div, mul);
}
"""
RUN = C.CFUNCTYPE(C.c_int, C.c_int, C.c_int, C.POINTER(C.c_float))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("handoff")
    (d / "h.cpp").write_text(SRC)
    so = str(d / "h.so")
    subprocess.run([os.environ.get("CXX", "g++"), "-O1", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "hawaiihybrid_b200", "csrc"), "-o", so, str(d / "h.cpp")], check=True)
    return C.CDLL(so)


def _pick(lib, default, times, fail_at=None):
    """times: {(div, mul): ms}; returns (rc, div, mul, thresholds timed)"""
    seen = []

    def run(d, m, ms):
        seen.append((d, m))
        if (d, m) == fail_at:
            return -3
        ms[0] = times[d, m]
        return 0

    d, m = C.c_int(), C.c_int()
    rc = lib.pick(default, RUN(run), C.byref(d), C.byref(m))
    return rc, d.value, m.value, seen


ALL = [(1, 8), (1, 4), (1, 2), (1, 1), (2, 1), (4, 1)]


@pytest.mark.parametrize("default", [1, 4, 8])
@pytest.mark.parametrize("noise", [(0, 0, 0, 0, 0, 0), (.01, 0, -.01, .01, -.01, 0), (-.01, .005, -.01, 0, .01, -.01)])
def test_noise_leaves_the_default(lib, default, noise):
    times = {k: 50.0 * (1.0 + e) for k, e in zip(ALL, noise)}
    rc, d, m, seen = _pick(lib, default, times)
    assert (rc, d, m) == (0, 1, default)
    assert len(seen) <= 3 and len(set(seen)) == len(seen)


@pytest.mark.parametrize("default,times,want", [
    (4, dict(zip(ALL, (40, 50, 60, 70, 80, 90))), (1, 8)),
    (4, dict(zip(ALL, (60, 50, 45, 40, 45, 50))), (1, 1)),
    (4, dict(zip(ALL, (60, 50, 45, 40, 35, 30))), (4, 1)),
    (4, dict(zip(ALL, (60, 50, 45, 60, 35, 30))), (1, 2)),
    (8, dict(zip(ALL, (60, 50, 45, 40, 41, 42))), (1, 1)),
    (1, dict(zip(ALL, (40, 44, 47, 50, 45, 40))), (1, 8)),
    (1, dict(zip(ALL, (70, 60, 55, 50, 45, 44.9))), (2, 1)),
])
def test_clear_gains_are_taken(lib, default, times, want):
    rc, d, m, _ = _pick(lib, default, times)
    assert (rc, d, m) == (0, *want)


def test_an_error_ends_the_choice(lib):
    times = dict.fromkeys(ALL, 50.0)
    assert _pick(lib, 4, times, fail_at=(1, 4))[0] == -3
    assert _pick(lib, 4, times, fail_at=(1, 8))[0] == -3
