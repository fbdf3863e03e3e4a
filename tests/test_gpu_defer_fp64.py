"""Deferred sample evaluation of the FP64 path (CO2-Ar: per-lane surface; N2-Ar: the dipole
network of 32 samples at once on the FP64 matrix instruction) against the in-kernel
placement on the same trajectories: the same steps, samples and statuses, C(t) equal up to
the order of the FP64 sums (every sample agrees to a few ulps, so 1e-12 of C(0) is several
hundred times their rounding), whole and in parts of an iteration, with failed trajectories
and at the shortest windows."""
import os

import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import lib_params, lib_system, oracle_params, oracle_system, rel_to_c0

pytestmark = pytest.mark.gpu
STAT_KEYS = ("n_steps", "n_rejected_steps", "n_rhs", "n_samples", "n_dense", "n_failed")


def _both(fn):
    from hawaiihybrid_b200 import _lib
    prev = _lib.defer_samples(-1)
    try:
        _lib.defer_samples(0)
        a = fn()
        _lib.defer_samples(1)
        b = fn()
    finally:
        _lib.defer_samples(prev)
    return a, b


@pytest.mark.parametrize("name", ["co2ar", "n2ar"])
@pytest.mark.parametrize("n,N", [(1500, 2048), (37, 700), (3, 1), (5, 2), (33, 3)])
def test_fp64_deferred_matches_in_kernel(name, n, N):
    import hawaiihybrid_b200 as hh
    ms = lib_system(name, 5)
    qp, _ = O.sample(5, oracle_system(name), oracle_params(name, N, 100.0), 300.0, n)
    p = lib_params(name, N, 100.0)
    (ca, sa), (cb, sb) = _both(lambda: hh.correlation_from_initial_conditions(ms, p, qp))
    assert rel_to_c0(cb, ca) < 1e-12
    for k in STAT_KEYS:
        assert getattr(sa, k) == getattr(sb, k), k
    assert list(sa.status) == list(sb.status)


@pytest.mark.parametrize("name", ["co2ar", "n2ar"])
def test_fp64_deferred_failure_and_parts(name):
    """A hard failure injected at one sample, and a context budget that splits each of the
    three iterations of a call into several launches."""
    import hawaiihybrid_b200 as hh
    from hawaiihybrid_b200 import _lib, hawaii
    lib = _lib.load()
    ms = lib_system(name, 7)
    p = lib_params(name, 600, 100.0)
    assert lib.hh_cuda_debug_inject(405, 1, 2, 5) == 0
    try:
        (ca, _, sa), (cb, _, sb) = _both(lambda: hawaii.correlation_iterations(ms, p, 300.0, 400, 3, seed=7))
        os.environ["HH_DEFER_BUDGET_MB"] = "1"  # about 100 trajectories a launch
        try:
            cc, _, sc = hawaii.correlation_iterations(ms, p, 300.0, 400, 3, seed=7)
        finally:
            del os.environ["HH_DEFER_BUDGET_MB"]
    finally:
        lib.hh_cuda_debug_inject(-1, 0, 0, 0)
    assert sa.n_failed == sb.n_failed == sc.n_failed == 1
    for i in range(3):
        assert rel_to_c0(cb[i], ca[i]) < 1e-12
        assert rel_to_c0(cc[i], ca[i]) < 1e-12
    # (the deferred branch of the failed trajectory is integrated to its end, in parts or not)
    assert sc.n_steps == sb.n_steps and sc.n_kernel_launches > sb.n_kernel_launches
