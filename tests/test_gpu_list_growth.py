"""Row capacities of the stored list and its sub-lists: sized for the mean
density, grown where a spot is denser, and no larger than what they hold."""
import dataclasses

import numpy as np
import pytest

from gpu_util import cpu, engine_for, rel_err, water_cluster

pytestmark = pytest.mark.gpu
FIELD_RTOL = 5e-5  # the field tolerance of the other GPU tests


def _first(capacity, n, volume, radius, factor):
    e = n / volume * 4 / 3 * np.pi * radius**3 * factor + 32
    return capacity if e >= capacity else (int(e) + 31) // 32 * 32


def _most(x, radius, box):
    d = x[:, None] - x[None]
    if box is not None:
        d -= np.asarray(box) * np.round(d / np.asarray(box))
    return int(((d * d).sum(-1) <= radius**2).sum(1).max()) - 3  # itself and its molecule


def _clump(tg, kind):
    """A system with a denser spot than its lists are first sized for."""
    if kind == "cells":  # the box of a liquid in the corner of one of eight times the volume: every list is too short
        s = tg.systems.make_config("water648", vdw=True)
        s.box = [2 * float(b) for b in s.box]
        assert _most(s.xyz, 9.0, s.box) > _first(10**6, s.n, np.prod(s.box), 9.0, 1.5)
    elif kind == "all pairs":  # rows of every atom, too short a cutoff sub-list
        w = tg.systems.make_config("water648")
        na = 300
        keep = (w.excl_ik < na).all(1)
        s = dataclasses.replace(w, xyz=w.xyz[:na].copy(), types=w.types[:na], frames=w.frames[:na].copy(), pole=w.pole[:na],
                                polarity=w.polarity[:na], thole=w.thole[:na], pdamp=w.pdamp[:na], excl_ik=w.excl_ik[keep],
                                excl_scale=w.excl_scale[keep], box=[22.0] * 3, mol_start=None, mol_size=None)
        s.settings = dict(w.settings)
        assert _most(s.xyz, 7.0, s.box) > _first(320, s.n, 22.0**3, 7.0, 1.5)
    else:  # two droplets far apart: too short a preconditioner sub-list
        s = water_cluster(tg, 216)
        s.xyz = np.concatenate([s.xyz[:324], s.xyz[:324] + 200.0])
        assert _most(s.xyz, 6.5, None) > _first(s.n, s.n, np.prod(np.ptp(s.xyz, axis=0)), 6.5, 3.0)
    return s


@pytest.mark.parametrize("kind", ["cells", "all pairs", "droplets"])
@pytest.mark.parametrize("first", ["field", "precond", "energy", "grad", "solve", "host solve", "staged"])
def test_lists_grow(gpu_lib, oracle, tg, kind, first):
    import torch

    s = _clump(tg, kind)
    e, o = engine_for(s), oracle.OracleSystem(s)
    rng = np.random.default_rng(4)
    u, up = rng.normal(size=(s.n, 3)) * 0.05, rng.normal(size=(s.n, 3)) * 0.05
    if first == "host solve":
        e.use_graph(False)
    if first == "staged":
        e.pair_lanes(8)
        e.pair_staging(True)
    calls = {"field": lambda: e.dfield() + e.ufield(u, up), "precond": lambda: e.sparse_precond(u, up),
             "energy": lambda: [torch.tensor(e.empole_energy()[1])], "grad": lambda: [e.emplar(gpu_lib.CALC_GRAD)[1]],
             "solve": lambda: e.induce()[:2]}
    call = calls["solve" if first in ("host solve", "staged") else first]
    a = [cpu(x) for x in call()]
    torch.cuda.synchronize()
    b = [cpu(x) for x in call()]  # on lists that are long enough
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
    for x, y in zip(calls["field"]() + calls["precond"](), o.dfield() + o.ufield(u, up) + o.sparse_precond(u, up)):
        assert rel_err(cpu(x), y) < FIELD_RTOL
    ref = o.induce()[:2]
    for x, y in zip(calls["solve"](), ref):  # both solved to 1e-6 D rms
        assert np.abs(cpu(x) - y).max() * tg.units.DEBYE < 2e-5


def test_hal_grows(gpu_lib, tg):
    s = _clump(tg, "cells")
    e = engine_for(s)
    a = e.ehal()
    b = e.ehal()
    assert a[0] == b[0] and np.array_equal(cpu(a[1]), cpu(b[1]))


def test_list_memory(gpu_lib, tg):
    """The sub-lists and their factors take the room of the pairs within
    their cutoffs: with the stored rows' capacity a liquid box with the van der
    Waals term took 44 bytes for each of its entries; half of that, and 120 MB
    for all else at this size, is more than enough."""
    import torch

    s = tg.systems.make_config("water12288", vdw=True)
    engine_for(s).ehal()  # the kernels are loaded
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    e = engine_for(s)
    e.ehal()
    torch.cuda.synchronize()
    used = free - torch.cuda.mem_get_info()[0]
    cap = e.list_stats()["capacity"]
    print(f"{used / 1e6:.0f} MB, stored rows of {cap}")
    assert used < 22 * cap * s.n + 120e6
