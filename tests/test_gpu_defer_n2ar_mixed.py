"""Mixed N2-Ar calls on both sides of the rule that defers their samples (2^19 sample times):
the default placement against samples in the trajectory kernel, and with a context budget
that splits the call's iterations into parts.  The same steps and samples; the dipole of a
sample is the same table lookup in both, so C(t) agrees up to the order of the FP64 sums
(1e-12 of C(0), the bound of the other placement tests)."""
import os

import numpy as np
import pytest

from tests.helpers import lib_params, lib_system, rel_to_c0

pytestmark = pytest.mark.gpu
STAT_KEYS = ("n_steps", "n_rejected_steps", "n_rhs", "n_samples", "n_dense", "n_failed")


@pytest.mark.parametrize("n,N,iters", [(64, 2048, 1), (511, 1024, 1), (512, 1024, 1), (700, 900, 2)])
@pytest.mark.parametrize("budget", [None, "1"])
def test_default_placement_matches_in_kernel(n, N, iters, budget):
    import hawaiihybrid_b200 as hh
    from hawaiihybrid_b200 import _lib, hawaii
    ms = lib_system("n2ar", 21)
    p = lib_params("n2ar", N, 100.0, mixed_tol=3e-8)
    run = lambda: hawaii.correlation_iterations(ms, p, 250.0, n, iters, hh.PRECISION_MIXED, seed=21)
    prev = _lib.defer_samples(-1)
    try:
        _lib.defer_samples(0)
        ca, na, sa = run()
        _lib.defer_samples(1)
        if budget:
            os.environ["HH_DEFER_BUDGET_MB"] = budget
        cb, nb, sb = run()
    finally:
        os.environ.pop("HH_DEFER_BUDGET_MB", None)
        _lib.defer_samples(prev)
    for k in STAT_KEYS:
        assert getattr(sa, k) == getattr(sb, k), k
    assert list(sa.status) == list(sb.status)
    np.testing.assert_array_equal(na, nb)
    for i in range(iters):
        assert rel_to_c0(cb[i], ca[i]) < 1e-12
