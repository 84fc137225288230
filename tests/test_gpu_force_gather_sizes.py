"""The reciprocal force gathers on both sides of every size at which they take
another number of atoms a warp (one up to 6,144 atoms, four up to 24,576, then
eight), with and without a part-filled last warp, against the FP64 gradient,
for the multipoles alone and with the induced dipoles."""
import numpy as np
import pytest

from gpu_util import cpu, engine_for

pytestmark = pytest.mark.gpu
GRAD_TOL = 2e-3  # as the other gradient tests, kcal/mol/A


@pytest.mark.parametrize("sites", [216, 217, 2048, 2049, 2051, 8192])
def test_force_gathers(gpu_lib, oracle, tg, sites):
    import torch

    nside = max(6, int(np.ceil(sites ** (1 / 3) - 1e-9)))
    nfft = next(n for n in (24, 30, 36, 40, 48, 54, 60, 64, 72, 80) if n >= 1.2 * 3.1 * nside)
    s = tg.systems.make_config("water648", nside=nside, box=3.1 * nside, n_sites=sites, nfft=nfft)
    e = engine_for(s)
    atom = [s.n - 1]
    gm = e.empole(gpu_lib.CALC_GRAD)[1]
    g = e.emplar(gpu_lib.CALC_GRAD)[1]
    gv = e.emplar(gpu_lib.CALC_GRAD | gpu_lib.CALC_VIRIAL)[1]  # both halves in order, on one grid
    torch.cuda.synchronize()
    om = oracle.empole_gradient_fd(s, atoms=atom)
    assert np.abs(cpu(gm)[atom] - om).max() < GRAD_TOL
    u, up = (cpu(x) for x in e.uind()[:2])
    o = om + oracle.epolar_gradient_fd(s, u, up, atoms=atom)
    assert np.abs(cpu(g)[atom] - o).max() < GRAD_TOL
    assert np.abs(cpu(gv)[atom] - o).max() < GRAD_TOL
