"""The sampler's fast paths against the oracle's sequential stream and rejection loop: stream
lengths around a word step (227), a block (624), the two-step turn and the segment
threshold; the CH4-CO2 rejection ahead of the momenta at temperatures whose acceptance runs
from one in thousands to most, for every pair state.  The words, the candidate counts and
which candidates are accepted are exact; the phase points agree to the rounding of the
device's transcendental functions (1e-12, as tests/test_gpu_ch4co2.py has it)."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import lib_params, lib_system, oracle_params, oracle_system

pytestmark = pytest.mark.gpu
SEG = 512 * 624


@pytest.mark.parametrize("n", [1, 226, 227, 228, 453, 454, 455, 623, 624, 625, 1248, 100_001, 2 * SEG - 625,
                               2 * SEG - 624, 2 * SEG + 1, 3 * SEG + 17, 33 * SEG, 34 * SEG + 5])
def test_mt_stream_lengths(n):
    from hawaiihybrid_b200 import _lib
    lib_system("hear")
    out = np.empty(n, dtype=np.uint32)
    _lib.check(_lib.load().hh_cuda_mt_stream(20240607, n, out))
    np.testing.assert_array_equal(out, O.mt_stream(20240607, n))


@pytest.mark.parametrize("T,ps,n", [(60.0, 1, 60), (100.0, 1, 700), (100.0, 2, 40), (150.0, 3, 500), (400.0, 1, 3000),
                                    (3000.0, 1, 3000)])
def test_ch4co2_candidates_match_oracle(T, ps, n):
    import hawaiihybrid_b200 as hh
    seed = 77
    ms = lib_system("ch4co2", seed)
    ref, nc = O.sample(seed, oracle_system("ch4co2"), oracle_params("ch4co2", 21, 200.0, ps=ps), T, n)
    qp, ng = hh.sample_initial_conditions(ms, lib_params("ch4co2", 21, 200.0, ps=ps), T, n, seed=seed)
    assert ng == int(nc)
    np.testing.assert_allclose(qp, ref, rtol=1e-12, atol=1e-12 * np.abs(ref).max())
