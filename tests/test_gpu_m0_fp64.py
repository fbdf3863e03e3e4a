"""The FP64 zeroth-moment kernel (a warp's samples against the temperatures, one temperature
per lane) against the oracle: every width of its temperature groups, the second chunk of 16,
sample counts around a warp, a block and the grid, and the three pair states.  The sums are
of positive terms whose error is that of V / kT (below 1e3) and of exp: 1e-12 at most, and
the bound is the 1e-10 of the other moment tests; the error estimate is the root of a
difference of such sums (1e-8)."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import lib_params, lib_system, oracle_params, oracle_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["hear", "co2ar", "n2ar"])
@pytest.mark.parametrize("nT,n,ps", [(1, 1, 1), (1, 33, 1), (2, 31, 3), (3, 257, 1), (4, 256, 1), (5, 1000, 3), (8, 4097, 2),
                                     (9, 113_663, 1), (15, 113_665, 3), (16, 32, 1), (17, 75_777, 1), (33, 999, 2)])
def test_m0_fp64_shapes(name, nT, n, ps):
    import hawaiihybrid_b200 as hh
    from hawaiihybrid_b200 import hawaii as H
    ms = lib_system(name)
    T = np.linspace(90.0, 700.0, nT)
    m, e = hh.calculate_m0(ms, lib_params(name, 64, 100.0, ps=ps), T, n, seed=1234567890123)
    op = oracle_params(name, 64, 100.0, ps=ps)
    ws, wq = O.m0(oracle_system(name), op, T, n, 1234567890123)
    mref, eref = H.moment_from_sums(ws, wq, n, O.m0_scale(op))
    np.testing.assert_allclose(m, mref, rtol=1e-10)
    if n > 1:
        np.testing.assert_allclose(e, eref, rtol=1e-8)
