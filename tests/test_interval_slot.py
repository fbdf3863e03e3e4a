"""The slot of a distance in the sample kernels' interval table (csrc/hh_interval.h), compiled
for the host: in range for every distance and for a NaN, which a double-to-int conversion
turns into INT_MIN; for finite distances the floor of 4 R, at most the last slot."""
import ctypes as C
import math
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = """
#include "hh_interval.h"
extern "C" int slot_d(double R) { return hh::r_slot<double>(R); }
extern "C" int slot_f(float R) { return hh::r_slot<float>(R); }
extern "C" int slots() { return hh::R_SLOTS; }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("slot")
    (d / "slot.cpp").write_text(SRC)
    so = str(d / "slot.so")
    subprocess.run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "hawaiihybrid_b200", "csrc"), "-o", so, str(d / "slot.cpp")], check=True)
    L = C.CDLL(so)
    L.slot_d.argtypes = [C.c_double]
    L.slot_f.argtypes = [C.c_float]
    return L


@pytest.mark.parametrize("R", [math.nan, -math.nan, math.inf, 1e300, 1e38, 3e9, 40.75, 41.0, 0.0, 5e-324])
def test_any_distance_stays_in_the_table(lib, R):
    n = lib.slots()
    assert 0 <= lib.slot_d(R) < n
    assert 0 <= lib.slot_f(R if abs(R) < 3e38 or R != R else math.inf) < n


def test_finite_distances_take_the_floor_of_four_r(lib):
    edges = np.arange(0, 168) / 4.0
    for R in np.concatenate([edges, np.nextafter(edges, 0.0), np.nextafter(edges, 50.0), np.linspace(0, 45, 997)]):
        want = min(int(math.floor(4.0 * R)), lib.slots() - 1)
        assert lib.slot_d(float(R)) == want
        f = np.float32(R)
        assert lib.slot_f(float(f)) == min(int(math.floor(4.0 * float(f))), lib.slots() - 1)
