"""Hand-off thresholds of several items per solo warp slot, fixed through the knob: every
multiple integrates the same steps (the item trace) and gives the same C(t) to the order of
the FP64 sums (1e-12 of C(0)); a pick that is read back and set again is the same pick; the
environment's threshold holds for small launches too, as the launch count shows."""
import numpy as np
import pytest

from tests.helpers import lib_params, lib_system, rel_to_c0

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,precision", [("hear", 0), ("hear", 1), ("co2ar", 0), ("co2ar", 1), ("n2ar", 0), ("n2ar", 1)])
def test_multiples_follow_the_same_steps(monkeypatch, name, precision):
    import hawaiihybrid_b200 as hh
    from hawaiihybrid_b200 import _lib
    L = _lib.load()
    ms = lib_system(name, 61)
    p = lib_params(name, 256, 100.0, mixed_tol=3e-8)
    qp, _ = hh.sample_initial_conditions(ms, p, 300.0, 9001, seed=61)

    def traced(q):
        tr = np.zeros(4 * 2 * len(q), dtype=np.uint32)
        assert L.hh_cuda_debug_item_trace(tr.ctypes.data, tr.size) == 0
        c, s = hh.correlation_from_initial_conditions(ms, p, q, precision)
        return tr.reshape(-1, 4)[:, 0].copy(), c, s.n_kernel_launches

    _lib.traj_tuning(precision, -1, -1)
    assert _lib.traj_handoff_mul(precision) == 0
    runs = {}
    for m in (1, 2, 4, 8):
        assert _lib.traj_handoff_mul(precision, m) == m
        assert _lib.traj_tuning(precision)[1] == 1 and _lib.traj_handoff_mul(precision) == m
        runs[m] = traced(qp)
    _lib.traj_tuning(precision, -1, -1)
    runs["tuned"] = traced(qp)
    w, d = _lib.traj_tuning(precision)
    m = _lib.traj_handoff_mul(precision)
    assert m in (1, 2, 4, 8) and d in (1, 2, 4) and (m == 1 or d == 1)
    _lib.traj_tuning(precision, -1, -1)
    _lib.traj_tuning(precision, w, d)
    if m > 1:
        _lib.traj_handoff_mul(precision, m)
    assert (_lib.traj_tuning(precision), _lib.traj_handoff_mul(precision)) == ((w, d), m)
    runs["again"] = traced(qp)
    for key, (s, c, _) in runs.items():
        np.testing.assert_array_equal(s, runs[1][0], err_msg=str(key))
        assert rel_to_c0(c, runs[1][1]) < 1e-12, key
    # 3,000 items: below the default threshold, above one item per slot
    _lib.traj_tuning(precision, -1, -1)
    free = traced(qp[:1500])[2]
    _lib.traj_tuning(precision, 0, 1)
    fixed = traced(qp[:1500])[2]
    _lib.traj_tuning(precision, -1, -1)
    monkeypatch.setenv("HH_TRAJ_HANDOFF_DIV", "1")
    assert traced(qp[:1500])[2] == fixed > free
    _lib.traj_tuning(precision, -1, -1)


def test_refused_multiples():
    from hawaiihybrid_b200 import _lib
    lib_system("hear", 1)
    for m in (-1, 3, 16):
        assert _lib.load().hh_cuda_debug_traj_handoff(0, m, None) != 0
    assert _lib.load().hh_cuda_debug_traj_handoff(7, 1, None) != 0
