"""Calls with short and long windows in turn, and bound pairs, whose trajectories fill the
window with steps: no call is repeated because its sample contexts overflow a buffer sized
for calls of another kind.  A repeated call launches every kernel twice, so the launch count
of the same call alone in a fresh context is the reference.  C(t) agrees to the order of the
FP64 sums (1e-12 of C(0), the bound of the other placement tests)."""
import pytest

from tests.helpers import lib_params, lib_system, rel_to_c0

pytestmark = pytest.mark.gpu


def _fresh(name):
    from hawaiihybrid_b200 import _lib
    _lib.load().hh_cuda_shutdown()
    return lib_system(name, 41)


@pytest.mark.parametrize("name,precision", [("co2ar", 0), ("co2ar", 1), ("n2ar", 0), ("n2ar", 1)])
def test_short_and_long_windows_in_turn(name, precision):
    import hawaiihybrid_b200 as hh
    n = 2500
    short, long_ = (lib_params(name, N, 100.0, mixed_tol=3e-8) for N in (40, 2048))
    ms = _fresh(name)
    qp, _ = hh.sample_initial_conditions(ms, long_, 300.0, n, seed=41)
    run = lambda p: hh.correlation_from_initial_conditions(ms, p, qp, precision)
    c0, s0 = run(long_)
    ms = _fresh(name)
    for _ in range(2):
        run(short)
        c, s = run(long_)
        assert s.n_kernel_launches == s0.n_kernel_launches
        assert s.n_steps == s0.n_steps and s.n_samples == s0.n_samples
        assert rel_to_c0(c, c0) < 1e-12


@pytest.mark.parametrize("name,precision", [("co2ar", 0), ("co2ar", 1), ("n2ar", 0), ("n2ar", 1)])
@pytest.mark.parametrize("N", [256, 4096])
def test_first_call_with_bound_pairs(name, precision, N):
    import hawaiihybrid_b200 as hh
    p = lib_params(name, N, 100.0, ps=2, mixed_tol=3e-8)
    ms = _fresh(name)
    qp, _ = hh.sample_initial_conditions(ms, p, 100.0, 2500, seed=41)
    c0, s0 = hh.correlation_from_initial_conditions(ms, p, qp, precision)
    c1, s1 = hh.correlation_from_initial_conditions(ms, p, qp, precision)
    assert s0.n_kernel_launches == s1.n_kernel_launches
    assert s0.n_steps == s1.n_steps and rel_to_c0(c1, c0) < 1e-12
