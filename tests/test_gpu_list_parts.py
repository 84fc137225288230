"""Calls form the parts of the per-step lists that they read: in every order
of the calls, at new positions and at the same ones, each gives the bits that
it gives alone."""
import itertools
import time

import numpy as np
import pytest

from gpu_util import cpu, engine_for

pytestmark = pytest.mark.gpu


def _calls(abi, e, u, up):
    return {
        "precond": lambda: e.sparse_precond(u, up),
        "ehal": lambda: e.ehal(),
        "energy": lambda: (e.empole_energy()[0],),
        "grad": lambda: e.empole(abi.CALC_GRAD | abi.CALC_VIRIAL)[1:],
        "field": lambda: e.dfield() + e.ufield(u, up),
        "solve": lambda: e.induce()[:2],
    }


def _bits(out):
    return [cpu(x) if hasattr(x, "detach") else np.asarray(x) for x in out]


@pytest.mark.parametrize("graph", [True, False])
def test_any_order_of_calls(gpu_lib, tg, graph):
    import torch

    s = tg.systems.make_config("water648", vdw=True)
    rng = np.random.default_rng(1)
    u, up = rng.normal(size=(s.n, 3)) * 0.05, rng.normal(size=(s.n, 3)) * 0.05
    frames = [torch.tensor(s.xyz + 0.05 * rng.normal(size=s.xyz.shape), dtype=torch.float32, device="cuda")
              for _ in range(2)]

    def engine():
        e = engine_for(s)
        e.use_graph(graph)
        e.ehal()  # the stored list, at the positions of the order
        return e

    def at(e, k):
        e.set_xyz_device(frames[k])
        e.mpole_init()

    names = list(_calls(gpu_lib, None, u, up))
    alone = {}
    for name, k in itertools.product(names, (0, 1)):
        e = engine()
        at(e, k)
        alone[name, k] = _bits(_calls(gpu_lib, e, u, up)[name]())
        torch.cuda.synchronize()
    e = engine()
    for turn in range(12):
        k = turn % 2
        at(e, k)
        for name in rng.permutation(names)[: 1 + turn % len(names)]:
            got = _bits(_calls(gpu_lib, e, u, up)[name]())
            torch.cuda.synchronize()
            for x, y in zip(got, alone[name, k]):
                assert np.array_equal(x, y), (turn, name)


def test_energies_pay_for_no_factors(gpu_lib, tg):
    """What a position update adds to the next call: a multipole energy reads
    one sub-list, a field every factor of it and of the preconditioner's, whose
    forming takes most of the refresh at this size."""
    import torch

    s = tg.systems.make_config("water98304")
    e = engine_for(s)
    u = np.zeros((s.n, 3))
    x = torch.tensor(s.xyz, dtype=torch.float32, device="cuda")

    def cost(call):
        def median(update):
            t = []
            for _ in range(30):
                if update:
                    e.set_xyz_device(x)
                torch.cuda.synchronize()
                t0 = time.perf_counter()
                call()
                torch.cuda.synchronize()
                t.append(time.perf_counter() - t0)
            return sorted(t)[len(t) // 2]

        return median(True) - median(False)

    energy, field = cost(e.empole_energy), cost(e.dfield)
    print(f"refresh before an energy {1e6 * energy:.0f} us, before a field {1e6 * field:.0f} us")
    assert energy < 0.8 * field
