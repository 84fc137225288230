"""A coordinate that is not a number reaches the van der Waals energy and
gradient: t9gb_set_xyz_device does not look at the coordinates, and the list
of the positions before stays in use, so the pairs themselves have to show it."""
import numpy as np
import pytest

from gpu_util import cpu, engine_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("atom", [0, 647])  # an oxygen; a hydrogen, whose site its oxygen's place enters
def test_broken_coordinate_is_not_dropped(gpu_lib, tg, atom, value):
    import torch

    s = tg.systems.make_config("water648", vdw=True)
    # the pairs within a molecule are scaled by zero: only those between molecules can show it
    assert len(s.vdw.scaled_v) == s.n and not s.vdw.scaled_v.any()
    e = engine_for(s)
    flags = gpu_lib.CALC_ENERGY | gpu_lib.CALC_GRAD
    assert np.isfinite(e.ehal(flags)[0])
    x = torch.tensor(np.asarray(s.xyz), dtype=torch.float32, device="cuda")
    x[atom, 1] = value
    e.set_xyz_device(x)
    en, g = e.ehal(flags)
    assert not np.isfinite(en)
    assert not np.isfinite(cpu(g)[atom]).all()
