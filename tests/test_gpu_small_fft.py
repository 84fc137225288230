"""The one-cluster PME transform of small cubic grids: every edge that has a
kernel, against the FP64 oracle and against cuFFT on the same system.  The
edges cover two to three planes and 16 to 100 columns a CTA, with and without
remainders over the cluster, and every pair of factors."""
import numpy as np
import pytest

from gpu_util import cpu, engine_for, rel_err

pytestmark = pytest.mark.gpu
FIELD_RTOL = 5e-5  # the field tolerance of the other GPU tests
SAME_RTOL = 2e-6  # two FP32 transforms of one grid


@pytest.mark.parametrize("n", [16, 18, 20, 24, 30, 32, 36, 40])
def test_small_grid_fields(gpu_lib, oracle, tg, n):
    s = tg.systems.make_config("water648", nfft=n)
    a, b = engine_for(s), engine_for(s)
    b.pme_own_fft(False)
    o = oracle.OracleSystem(s)
    rng = np.random.default_rng(n)
    u, up = rng.normal(size=(s.n, 3)) * 0.05, rng.normal(size=(s.n, 3)) * 0.05
    for _ in range(2):  # the second pass reads the grid that the first one cleared
        for x, y, r in zip(a.dfield() + a.ufield(u, up), b.dfield() + b.ufield(u, up), o.dfield() + o.ufield(u, up)):
            assert rel_err(cpu(x), cpu(y)) < SAME_RTOL
            assert rel_err(cpu(x), r) < FIELD_RTOL
    # the dipole grid beside the permanent one
    abi = gpu_lib
    ga, gb = a.emplar(abi.CALC_ENERGY | abi.CALC_GRAD)[1], b.emplar(abi.CALC_ENERGY | abi.CALC_GRAD)[1]
    assert rel_err(cpu(ga), cpu(gb)) < 1e-5
    assert a.stats()[0] == b.stats()[0]
