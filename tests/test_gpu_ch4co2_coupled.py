"""The coupled-form FP64 CH4-CO2 dipole kernel (its own frame, rotated invariants and
Legendre sums) against the entry-stream kernel of the same reference tables: ensembles of
sizes around a warp task, and single configurations where its frame degenerates (CO2 along,
against and almost along the intermolecular axis, and across it) in every radial piece.

Tolerances: both kernels sum about 1e4 terms of the size of the dipole's scale with a few
digits of cancellation, so they agree to 1e4 x 10 x 1.1e-16 = 1e-11 of the scale at that R;
an ensemble's C(t) averages that below 1e-12 of C(0)."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import lib_params, lib_system, oracle_params, oracle_system, rel_to_c0

pytestmark = pytest.mark.gpu
ENTRIES, COUPLED = 1, -2


def _with(variant, fn):
    from hawaiihybrid_b200 import _lib
    L = _lib.load()
    _lib.check(L.hh_cuda_debug_set_ch4_dipole(0, variant))
    try:
        return fn()
    finally:
        _lib.check(L.hh_cuda_debug_set_ch4_dipole(0, 0))


@pytest.mark.parametrize("n", [1, 31, 33, 400])
def test_coupled_ensemble_matches_entry_stream(n):
    import hawaiihybrid_b200 as hh
    ms = lib_system("ch4co2")
    p = lib_params("ch4co2", 21, 200.0)
    qp, _ = O.sample(11, oracle_system("ch4co2"), oracle_params("ch4co2", 21, 200.0), 250.0, n)
    a, b = (_with(v, lambda: hh.correlation_from_initial_conditions(ms, p, qp)[0]) for v in (ENTRIES, COUPLED))
    assert rel_to_c0(b, a) < 1e-12


@pytest.mark.parametrize("R", [4.6, 5.1, 6.3, 7.9, 9.4, 9.75, 10.25, 11.5, 13.0, 17.0, 22.0, 27.0, 33.0])
def test_coupled_at_degenerate_angles(R):
    """|mu0|^2 = C(0) of one configuration (N = 1)."""
    import hawaiihybrid_b200 as hh
    ms = lib_system("ch4co2")
    p = lib_params("ch4co2", 1, 200.0)
    rng = np.random.default_rng(3)
    got = []
    for eps in (0.0, 1e-13, 1e-9, 1e-5, 0.3, np.pi / 2, np.pi - 1e-9, np.pi):
        Phi, Th = rng.uniform(0, 2 * np.pi), rng.uniform(0.8, 1.2)
        qp = np.array([Phi, 1.0, Th, 1.0, R, -1.0, rng.uniform(0, 6), 1.0, rng.uniform(0.4, 2.5), 1.0,
                       rng.uniform(0, 6), 1.0, Phi, 1.0, Th + eps, 1.0])
        got.append([_with(v, lambda: hh.correlation_from_initial_conditions(ms, p, qp)[0][0]) for v in (ENTRIES, COUPLED)])
    got = np.array(got)
    assert np.all(got > 0.0)
    np.testing.assert_allclose(got[:, 1], got[:, 0], rtol=0, atol=1e-11 * got[:, 0].max())
