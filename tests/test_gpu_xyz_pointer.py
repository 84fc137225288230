"""t9gb_set_xyz_device takes coordinates from wherever a device-to-device copy
does: the GPU's own memory is read by the kernel that sorts the positions, any
other (here pinned host memory) is copied first."""
import ctypes as C

import numpy as np
import pytest

from gpu_util import cpu, engine_for

pytestmark = pytest.mark.gpu


def test_memory_kinds(gpu_lib, tg):
    import torch

    s = tg.systems.make_config("water648")
    e = engine_for(s)
    rng = np.random.default_rng(2)
    x = torch.tensor(s.xyz + 0.05 * rng.normal(size=s.xyz.shape), dtype=torch.float32)
    e.set_xyz(x.double().numpy())
    e.mpole_init()
    want = [cpu(v) for v in e.induce()[:2]]
    odd = torch.zeros(3 * s.n + 1, device="cuda")[1:].view(s.n, 3)  # four bytes off an allocation's start
    odd.copy_(x)
    for t in (x.cuda(), odd, x.pin_memory()):
        e.set_xyz(s.xyz)
        e.set_xyz_device(t)
        e.mpole_init()
        for a, b in zip(e.induce()[:2], want):
            assert np.array_equal(cpu(a), b)


def test_null_pointer(gpu_lib, tg):
    e = engine_for(tg.systems.make_config("water648"))
    assert e.lib.t9gb_set_xyz_device(e.h, C.c_void_p(0)) == gpu_lib.T9GB_BAD_ARG
