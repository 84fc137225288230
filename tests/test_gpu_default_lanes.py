"""The default lanes per atom of the field and force kernels, on both sides
of every size at which they change, against one choice for all sizes.  The
two differ in the order in which a row's FP32 terms are added: some 150 terms
of either sign, each rounded to 6e-8, and a solve that both end below the same
residual."""
import pytest

from gpu_util import cpu, engine_for, rel_err

pytestmark = pytest.mark.gpu
RTOL = 1e-5


@pytest.mark.parametrize("nside, sites", [(7, 256), (7, 267), (10, 768), (10, 779), (11, 1024), (11, 1035)])
def test_default_lanes(gpu_lib, tg, nside, sites):
    s = tg.systems.make_config("water648", nside=nside, box=3.1 * nside, n_sites=sites, nfft=40)
    a, b = engine_for(s), engine_for(s)
    b.pair_lanes(8)
    b.force_lanes(4)
    ga, gb = (e.emplar(gpu_lib.CALC_ENERGY | gpu_lib.CALC_GRAD)[1] for e in (a, b))
    assert rel_err(cpu(ga), cpu(gb)) < RTOL
    assert a.stats()[0] == b.stats()[0]
    for x, y in zip(a.induce()[:2] + a.dfield(), b.induce()[:2] + b.dfield()):
        assert rel_err(cpu(x), cpu(y)) < RTOL


def test_learning_keeps_its_route(gpu_lib, tg):
    """While the learned guess trains, a small box solves as with the larger boxes' kernels, bit for bit."""
    s = tg.systems.make_config("water648")
    a, b = engine_for(s), engine_for(s)
    b.pair_lanes(8)
    b.pme_own_fft(False)
    for e in (a, b):
        e.learn_config(3)
    for _ in range(2):
        for x, y in zip(a.induce()[:2], b.induce()[:2]):
            assert (x == y).all()
    assert (a.learn_weights() == b.learn_weights()).all()
