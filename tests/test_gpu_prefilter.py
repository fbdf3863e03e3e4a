"""The CH4-CO2 rejection ahead of the momenta (an FP32 energy with a bound on its error)
against the FP64 decision, where it is closest: each candidate's last word is the largest
that FP64 still accepts, found by bisection, so that any error of the FP32 exponent beyond
its bound rejects a candidate that FP64 accepts.  Polar angles next to the poles (words near
0 and 2^32), phases next to a full turn, contact and far distances, low and high
temperatures.  The decisions are whole: no tolerance."""
import numpy as np
import pytest

from tests.helpers import RMIN_CH4CO2, lib_params, lib_system

pytestmark = pytest.mark.gpu
D = 25


def _accepted(p, T, w, prefilter):
    from hawaiihybrid_b200 import _lib
    return _lib.candidate_accepted(p, T, w, prefilter)


def _words(rng, n, R_hi):
    """n candidates at distances up to R_hi (of a range to 40 bohr)."""
    w = rng.integers(1, 1 << 32, size=(n, D), dtype=np.uint64)
    frac = (R_hi ** 3 - RMIN_CH4CO2 ** 3) / (40.0 ** 3 - RMIN_CH4CO2 ** 3)
    w[:, 0] = (rng.random(n) * frac * 4294967295.0).astype(np.uint64)
    # in three of four candidates some of the angles lie at a log-uniform distance from 0 or 2^32
    for col in range(1, 8):
        near = (2.0 ** rng.uniform(0.0, 31.0, n)).astype(np.uint64)
        end = np.where(rng.random(n) < 0.5, near, (1 << 32) - near)
        w[:, col] = np.where((np.arange(n) % 4 != 0) & (rng.random(n) < 0.5), end, w[:, col])
    return np.minimum(w, 0xFFFFFFFF).astype(np.uint32)


def test_candidate_beside_a_pole():
    p = lib_params("ch4co2", 21, 200.0, ps=3)
    lib_system("ch4co2", 1)
    w = np.full((1, D), 0x40000001, dtype=np.uint32)
    w[0, :8] = [11965176, 3904304333, 1157991612, 1738975247, 2104056694, 2523603405, 3919908914, 4294967181]
    w[0, 24] = 1669  # ln u = -14.7607; the FP64 weight is exp(-14.7508)
    assert _accepted(p, 100.0, w, False)[0]
    assert _accepted(p, 100.0, w, True)[0]


@pytest.mark.parametrize("T", [0.5, 5.0, 40.0, 100.0, 300.0, 3000.0])
@pytest.mark.parametrize("R_hi", [6.0, 9.0, 40.0])
def test_closest_decisions_agree(T, R_hi):
    n = 60_000
    p = lib_params("ch4co2", 21, 200.0, ps=3)
    lib_system("ch4co2", 1)
    w = _words(np.random.default_rng(int(10 * T + R_hi)), n, R_hi)
    lo, hi = np.zeros(n, dtype=np.uint64), np.full(n, 1 << 32, dtype=np.uint64)  # accepted at lo, not at hi
    for _ in range(32):
        mid = (lo + hi) // 2
        w[:, 24] = mid.astype(np.uint32)
        a = _accepted(p, T, w, False)
        lo, hi = np.where(a, mid, lo), np.where(a, hi, mid)
    w[:, 24] = lo.astype(np.uint32)
    a = _accepted(p, T, w, False)
    assert a[lo > 0].all()
    np.testing.assert_array_equal(_accepted(p, T, w, True), a)
    # and a word further, where FP64 rejects
    w[:, 24] = np.minimum(hi, 0xFFFFFFFF).astype(np.uint32)
    np.testing.assert_array_equal(_accepted(p, T, w, True), _accepted(p, T, w, False))
