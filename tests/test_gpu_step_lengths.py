"""The one-cluster vector steps of small boxes add p.Ap as the kernels of the
larger boxes do: 32 products in FP32, everything above in FP64.  The two then
differ in FP64 roundings alone, the step lengths, rounded to FP32, do not, and
whole solves agree bit for bit with those of the mask's bit 1, which has the
larger boxes' kernels at every size.  A thread has one product up to 682 slots, two
from there, five at 3,072."""
import numpy as np
import pytest

from gpu_util import engine_for, water_cluster

pytestmark = pytest.mark.gpu


def _same(s):
    a, b = engine_for(s), engine_for(s)
    b.pcg_fusion(3)
    for x, y in zip(a.induce()[:2], b.induce()[:2]):
        assert (x == y).all()


@pytest.mark.parametrize("sites", [216, 227, 455, 683, 1024])
def test_box(gpu_lib, tg, sites):
    nside = max(6, int(np.ceil(sites ** (1 / 3) - 1e-9)))
    _same(tg.systems.make_config("water648", nside=nside, box=3.1 * nside, n_sites=sites, nfft=40))


def test_cluster(gpu_lib, tg):
    _same(water_cluster(tg, 216))
