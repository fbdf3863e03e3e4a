"""Launches below the tuning threshold after a large, tuned one take the route they take
before it (the default hand-off threshold: all items in the solo kernel up to there), which
the number of kernel launches shows.  A threshold of one item per warp slot, fixed through
the tuning knob, holds for launches of every size."""
import pytest

from tests.helpers import lib_params, lib_system, rel_to_c0

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,precision", [("hear", 0), ("hear", 1), ("co2ar", 0), ("co2ar", 1), ("n2ar", 0), ("n2ar", 1)])
def test_small_launch_after_a_tuned_one(name, precision):
    import hawaiihybrid_b200 as hh
    from hawaiihybrid_b200 import _lib
    _lib.load().hh_cuda_shutdown()
    ms = lib_system(name, 51)
    p = lib_params(name, 512, 100.0, mixed_tol=3e-8)
    qp, _ = hh.sample_initial_conditions(ms, p, 300.0, 9000, seed=51)
    small = [qp[:k] for k in (1300, 2300, 4000)]
    run = lambda q: hh.correlation_from_initial_conditions(ms, p, q, precision)
    run(qp[:2000])                    # (buffers, context estimates)
    before = [run(q) for q in small]
    run(qp)                           # tunes
    assert _lib.traj_tuning(precision)[0] in (4, 8)
    for q, (c0, s0) in zip(small, before):
        c, s = run(q)
        assert s.n_kernel_launches == s0.n_kernel_launches, len(q)
        assert s.n_steps == s0.n_steps and rel_to_c0(c, c0) < 1e-12
    w, _ = _lib.traj_tuning(precision, 0, 1)
    c, s = run(small[2])
    assert s.n_kernel_launches > before[0][1].n_kernel_launches  # the bulk kernel, then the solo kernel
    assert s.n_steps == before[2][1].n_steps and rel_to_c0(c, before[2][0]) < 1e-12
    _lib.traj_tuning(precision, -1, -1)
