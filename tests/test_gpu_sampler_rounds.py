"""Small requests at a low acceptance (bound pairs): the candidates are tried in rounds of at
least 65,536 after the first, short one, so the number of launches follows the number of
candidates and not the size of the request.  A round is one candidate launch (two for CH4-CO2),
three of the compaction and at most seven of the stream; the trajectories of 16 phase points
take 32 launches at most."""
import pytest

from tests.helpers import lib_params, lib_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,T", [("hear", 300.0), ("co2ar", 300.0), ("n2ar", 300.0), ("ch4co2", 300.0), ("hear", 50.0)])
def test_rounds_follow_the_candidates(name, T):
    import hawaiihybrid_b200 as hh
    ms = lib_system(name, 7)
    p = lib_params(name, 16, 100.0, ps=2, mixed_tol=3e-8)
    for seed in (7, 8, 9):
        _, nc = hh.sample_initial_conditions(ms, p, T, 16, seed=seed)
        _, _, st = hh.correlation_iteration(ms, p, T, 16, seed=seed)
        rounds = 2 + nc // 65536
        assert st.n_kernel_launches <= 12 * rounds + 32, (seed, nc, st.n_kernel_launches)
