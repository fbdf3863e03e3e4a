"""Launches around the hand-off thresholds (148 SMs x warps per SM x 1, 4 and 8 items: all
items in the solo kernel up to there, the bulk kernel first above): a call equals the sum of
calls over its parts, which take other routes, to the order of the FP64 sums (1e-12 of C(0)),
with the same number of steps, since both kernels take the same ones."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import lib_params, lib_system, oracle_params, oracle_system, rel_to_c0

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,precision,n", [("hear", 0, 2369), ("hear", 1, 2400), ("co2ar", 0, 2369), ("co2ar", 1, 2369),
                                              ("n2ar", 0, 4737), ("n2ar", 1, 4800), ("n2ar", 0, 600)])
def test_call_equals_its_parts(name, precision, n):
    import hawaiihybrid_b200 as hh
    N, dt = 256, 100.0
    ms = lib_system(name, 3)
    qp, _ = O.sample(3, oracle_system(name), oracle_params(name, N, dt), 300.0, n)
    p = lib_params(name, N, dt, mixed_tol=3e-8)
    c, s = hh.correlation_from_initial_conditions(ms, p, qp, precision)
    parts = [hh.correlation_from_initial_conditions(ms, p, qp[a:a + n // 5 + 1], precision)
             for a in range(0, n, n // 5 + 1)]
    assert rel_to_c0(sum(q for q, _ in parts), c) < 1e-12
    assert sum(t.n_steps for _, t in parts) == s.n_steps
    assert sum(t.n_samples for _, t in parts) == s.n_samples
