"""The real-space rows, grid gathers and sums at the sizes where a kernel or
its shape changes, against the FP64 oracle."""
import numpy as np
import pytest

from gpu_util import cpu, engine_for, rel_err, water_cluster

pytestmark = pytest.mark.gpu
FIELD_RTOL = 5e-5  # the field tolerance of the other GPU tests


def _box(tg, sites, **kw):
    nside = max(6, int(np.ceil(sites ** (1 / 3) - 1e-9)))
    nfft = next(n for n in (24, 30, 36, 40, 48, 54, 60, 64, 72, 80, 90, 96, 100, 108) if n >= 1.2 * 3.1 * nside)
    return tg.systems.make_config("water648", nside=nside, box=3.1 * nside, n_sites=sites, nfft=nfft, **kw)


def _fields(e, o, n, precond=True):
    rng = np.random.default_rng(n)
    u, up = rng.normal(size=(n, 3)) * 0.05, rng.normal(size=(n, 3)) * 0.05
    got, ref = e.dfield() + e.ufield(u, up), o.dfield() + o.ufield(u, up)
    if precond:
        got, ref = got + e.sparse_precond(u, up), ref + o.sparse_precond(u, up)
    for x, y in zip(got, ref):
        assert rel_err(cpu(x), y) < FIELD_RTOL


# 810 molecules fill 152 half-SM blocks at eight lanes, 811 one more
@pytest.mark.parametrize("sites", [216, 217, 227, 810, 811])
def test_rows_of_every_lane_count(gpu_lib, oracle, tg, sites):
    s = _box(tg, sites)
    e, o = engine_for(s), oracle.OracleSystem(s)
    for lanes in (4, 32, 16, 8):  # each change lays the sub-lists out anew
        e.pair_lanes(lanes)
        _fields(e, o, s.n)


@pytest.mark.parametrize("nmol", [1, 10, 11, 40])
def test_rows_of_a_cluster(gpu_lib, oracle, tg, nmol):
    s = water_cluster(tg, nmol)
    e, o = engine_for(s), oracle.OracleSystem(s)
    for lanes in (4, 32, 16, 8):
        e.pair_lanes(lanes)
        _fields(e, o, s.n, precond=False)


@pytest.mark.parametrize("sites", [216, 227, 811])
def test_inner_rows(gpu_lib, oracle, tg, sites):
    """With the van der Waals cutoff the field rows are cut from a longer list."""
    s = _box(tg, sites, vdw=True)
    e, o = engine_for(s), oracle.OracleSystem(s)
    e.ehal()
    _fields(e, o, s.n)


# the spread forms the direction up to 4,096 slots (1,365 molecules)
@pytest.mark.parametrize("sites", [1365, 1366])
def test_direction_in_the_spread(gpu_lib, tg, sites):
    s = _box(tg, sites)
    a, b = engine_for(s), engine_for(s)
    b.lib.t9gb_set_pcg_fusion(b.h, 57)  # without the chain, the direction has its own kernel
    for x, y in zip(a.induce()[:2], b.induce()[:2]):
        assert rel_err(cpu(x), cpu(y)) < 1e-5  # both solved to 1e-5 D rms on dipoles of about 1 D
    assert a.stats()[0] == b.stats()[0]


# one cluster takes both vector steps up to 3,072 slots (1,024 molecules); bit
# 1 of the mask has its own pair of kernels at every size
@pytest.mark.parametrize("sites", [216, 227, 1024, 1025])
def test_vector_steps(gpu_lib, tg, sites):
    s = _box(tg, sites)
    a, b = engine_for(s), engine_for(s)
    b.lib.t9gb_set_pcg_fusion(b.h, 3)
    for x, y in zip(a.induce()[:2], b.induce()[:2]):
        assert rel_err(cpu(x), cpu(y)) < 1e-5
    assert a.stats()[0] == b.stats()[0]


@pytest.mark.parametrize("nmol", [1, 11, 40])
def test_vector_steps_of_a_cluster(gpu_lib, oracle, tg, nmol):
    s = water_cluster(tg, nmol)
    got, ref = engine_for(s).induce()[:2], oracle.OracleSystem(s).induce()[:2]
    for x, y in zip(got, ref):  # two solves to 1e-6 D rms
        assert np.abs(cpu(x) - y).max() * tg.units.DEBYE < 2e-5


# rows of 16 lanes below and of 8 above 32,768 atoms; queues that never fill
# (a few pairs) and that stay part full
@pytest.mark.parametrize("sites, vacuum", [(216, False), (227, False), (10923, False), (216, True)])
def test_hal_rows(gpu_lib, oracle, tg, sites, vacuum):
    from oracle import mm_oracle

    s = _box(tg, sites, vdw=True)
    if vacuum:  # molecules twice as far apart: most rows hold less than a chunk
        s.xyz = np.asarray(s.xyz) + np.repeat(np.asarray(s.xyz)[::3], 3, axis=0)
        s.box = [2 * float(b) for b in s.box]
    e = engine_for(s)
    en, g, _ = e.ehal(gpu_lib.CALC_ENERGY | gpu_lib.CALC_GRAD | gpu_lib.CALC_VIRIAL)
    if sites < 1000:
        eo = mm_oracle.hal_energy(s)
        assert abs(en - eo) < 2e-5 * abs(eo) + 1e-4
        atoms = [0, 1, s.n // 2, s.n - 1]
        go = oracle._fd(lambda x: mm_oracle.hal_energy(s, x), np.asarray(s.xyz, dtype=np.float64), atoms, 1e-5)
        assert np.abs(cpu(g)[atoms] - go).max() < 2e-4
    # no net force: each pair's two sides come from two rows
    g = cpu(g)
    assert np.abs(g.sum(0)).max() < 1e-5 * np.abs(g).sum(0).max()


# atoms per warp of the force gathers: four up to 24,576 atoms, eight above;
# a last warp that is full, or holds one molecule
@pytest.mark.parametrize("sites", [216, 217, 8193])
def test_force_gathers(gpu_lib, oracle, tg, sites):
    import torch

    s = _box(tg, sites)
    e = engine_for(s)
    _, g = e.emplar(gpu_lib.CALC_GRAD)[:2]
    torch.cuda.synchronize()  # without an energy or a virial the call does not wait for its stream
    u, up = (cpu(x) for x in e.uind()[:2])
    atoms = [0, s.n - 1] if sites < 1000 else [s.n - 1]
    go = oracle.empole_gradient_fd(s, atoms=atoms) + oracle.epolar_gradient_fd(s, u, up, atoms=atoms)
    assert np.abs(cpu(g)[atoms] - go).max() < 2e-3  # as the other gradient tests
