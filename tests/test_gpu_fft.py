"""The batched transform (hh_fft.cuh) through its three users, against the oracle: lengths of
one, two and three passes, every remainder of the radix-8 steps, the smallest lengths, and
(CF -> SF) both sides of the page-locked staging's limit.  The transform's error is a few
roundings per radix step of the largest term: 1e-12 of the peak, the bound of the other CF -> SF
test; the spectra and lagged sums carry the trajectories' 1e-8."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import lib_params, lib_system, oracle_params, oracle_system, rel_to_c0

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("logN", [0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 15, 16, 17, 18, 20, 21])
def test_idct_lengths(logN):
    import hawaiihybrid_b200 as hh
    lib_system("hear")
    N, dt = 1 << logN, 150.0
    rng = np.random.default_rng(logN)
    data = np.exp(-np.arange(N) / (0.1 * N)) * (1 + 0.01 * rng.standard_normal(N))
    t = dt * np.arange(max(N, 2))
    cf = hh.CFnc(t=t, data=data.copy(), ntraj=1.0, Temperature=300.0, normalized=True)
    sf = hh.idct_cf_to_sf(cf)
    nu_ref, sf_ref, cf_ref = O.idct_cf_to_sf(data, dt)
    assert np.max(np.abs(sf.data - sf_ref)) <= 1e-12 * np.max(np.abs(sf_ref))
    np.testing.assert_allclose(sf.nu, nu_ref, rtol=1e-12)
    np.testing.assert_allclose(cf.data, cf_ref, rtol=0, atol=1e-15)


def test_idct_nan_leaves_the_input():
    import hawaiihybrid_b200 as hh
    lib_system("hear")
    data = np.ones(2048)
    data[1999] = np.nan
    cf = hh.CFnc(t=np.arange(2048.0), data=data.copy(), ntraj=1.0, Temperature=300.0, normalized=True)
    with pytest.raises(hh.HHError):
        hh.idct_cf_to_sf(cf)
    np.testing.assert_array_equal(cf.data, data)


@pytest.mark.parametrize("N,dt,n", [(2, 200.0, 9), (4, 200.0, 5), (64, 200.0, 33), (128, 200.0, 8), (256, 200.0, 301),
                                    (512, 800.0, 2), (1024, 400.0, 1), (4096, 100.0, 7), (8192, 50.0, 7), (16384, 25.0, 4),
                                    (1 << 19, 0.8, 3)])
@pytest.mark.parametrize("trunc", [False, True])
def test_prmu_lengths(N, dt, n, trunc):
    import hawaiihybrid_b200 as hh
    name, T, seed = "hear", 300.0, 11
    ms = lib_system(name, seed)
    fmax = 0.9 / (2.99792458e10 * dt * 2.4188843265857e-17) / 2.0
    if N > 512:
        fmax = min(fmax, 700.0)
    _, sf, cnt, _ = hh.prmu_iteration(ms, lib_params(name, N, dt), T, 40.0, n, fmax, trunc, 0, seed=seed)
    ref, cnt_ref = O.prmu(oracle_system(name), oracle_params(name, N, dt), T, 40.0, n, sf.size, seed, allow_trunc=trunc)
    assert cnt == cnt_ref
    assert np.max(np.abs(sf - ref)) <= 1e-8 * np.max(np.abs(ref))


@pytest.mark.parametrize("N", [1, 2, 129, 3000])
def test_zimmermann_lengths(N):
    import hawaiihybrid_b200 as hh
    name, T, dt = "hear", 50.0, 200.0
    ms = lib_system(name)
    p = lib_params(name, N, dt, ps=2)
    p.use_zimmermann_trick = True
    op = oracle_params(name, N, dt, ps=O.PS_BOUND)
    qp, _ = O.sample(5, oracle_system(name), op, T, 7)
    crln, st = hh.correlation_from_initial_conditions(ms, p, qp)
    op.zimmermann = 1
    ref = O.correlation_sum(oracle_system(name), op, qp)
    assert st.n_failed == 0
    assert rel_to_c0(crln, ref) < 1e-8
