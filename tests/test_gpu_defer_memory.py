"""A call whose sample contexts cannot be allocated takes its samples in the trajectory
kernel, as it would without the sample kernels: the same C(t) (to the order of the FP64 sums;
mixed CO2-Ar to FP32 rounding, the bounds of the other placement tests) and statistics, no
error, and the next call defers again.  The estimate and the budget ask for more memory than
any device has, so the allocation is refused at once."""
import pytest

from tests.helpers import lib_params, lib_system, rel_to_c0

pytestmark = pytest.mark.gpu
STAT_KEYS = ("n_steps", "n_rejected_steps", "n_rhs", "n_samples", "n_dense", "n_failed")


@pytest.mark.parametrize("name,precision,tol", [("co2ar", 0, 1e-12), ("n2ar", 0, 1e-12), ("co2ar", 1, 1e-6),
                                                ("n2ar", 1, 1e-12)])
def test_no_memory_for_contexts(monkeypatch, name, precision, tol):
    import hawaiihybrid_b200 as hh
    from hawaiihybrid_b200 import _lib, hawaii
    ms = lib_system(name, 31)
    p = lib_params(name, 700, 100.0, mixed_tol=3e-8)
    run = lambda: hawaii.correlation_iterations(ms, p, 300.0, 1000, 1, precision, seed=31)
    prev = _lib.defer_samples(2)
    try:
        ca, _, sa = run()
        monkeypatch.setenv("HH_DEFER_EST", "1e6")          # 2,000 items: 0.4 to 0.8 TB
        monkeypatch.setenv("HH_DEFER_BUDGET_MB", "4e6")
        cb, _, sb = run()
        monkeypatch.delenv("HH_DEFER_EST")
        monkeypatch.delenv("HH_DEFER_BUDGET_MB")
        cc, _, sc = run()
    finally:
        _lib.defer_samples(prev)
    assert rel_to_c0(cb[0], ca[0]) < tol and rel_to_c0(cc[0], ca[0]) < 1e-12
    for k in STAT_KEYS:
        assert getattr(sa, k) == getattr(sb, k) == getattr(sc, k), k
    assert list(sa.status) == list(sb.status) == list(sc.status)
    assert sb.n_kernel_launches < sa.n_kernel_launches == sc.n_kernel_launches
