"""t9gb_ufield_noalloc over its sizes, against the same field in FP64.

The sizes lie at the edges of what a kernel stages (groups of 32 partners,
1,024 positions at a time, eight atoms a block); the atoms are in a random
order or along lines (bounding boxes that reach everything, or little), some
of them box lengths away from the first image.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
# FP32 pair terms (a few 1e-7 each) and 100 to 200 of them per atom added in
# FP32, of which about a tenth is left after cancellation
FIELD_RTOL = 2.0e-5
CUTOFF = 7.0


def _fp64(x, pd, th, u, box):
    """Field at every atom and whether one of its pairs lies at the cutoff's edge, by rows."""
    import torch

    f, edge = torch.zeros_like(x), torch.zeros(len(x), dtype=torch.bool, device=x.device)
    for a in range(0, len(x), 512):
        d = x[None] - x[a : a + 512, None]
        if box is not None:
            d = d - box * torch.round(d / box)
        r2 = (d * d).sum(-1)
        own = torch.arange(len(x), device=x.device)[None] == torch.arange(a, a + len(d), device=x.device)[:, None]
        use = (r2 <= CUTOFF**2) & ~own
        edge[a : a + 512] = ((r2 / CUTOFF**2 - 1).abs() < 1.0e-5).any(1)
        r = torch.where(use, r2, torch.ones_like(r2)).sqrt()
        au = torch.minimum(th[a : a + 512, None], th[None]) * (r / (pd[a : a + 512, None] * pd[None])) ** 3
        ex = torch.exp(-au)
        l3, l5 = (1 - ex) / r**3 * use, (1 - (1 + au) * ex) * 3 / r**5 * use
        f[a : a + 512] = torch.einsum("ij,ijk->ik", l5 * torch.einsum("ijk,jk->ij", d, u), d) - l3 @ u
    return f, edge


@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 1023, 1025, 2047, 2049, 4100, 8192])
@pytest.mark.parametrize("ordered, pbc, inplace", [(True, True, False), (False, True, True), (True, False, False)])
def test_noalloc_sizes(gpu_lib, n, ordered, pbc, inplace):
    import torch

    lib = gpu_lib.load()
    g = np.random.default_rng(n)
    side = max(16.0, (n / 0.1) ** (1 / 3))
    m = int(np.ceil(n ** (1 / 3)))
    x = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * (side / m)
    x = x + g.uniform(-0.2, 0.2, (n, 3)) * min(1.0, side / m)
    if not ordered:
        x = x[g.permutation(n)]
    box = np.array([side, side, 1.1 * side])
    if pbc:
        x = x + box * g.integers(-2, 3, (n, 3))
    t = [torch.tensor(v, dtype=torch.float32, device="cuda") for v in
         (x, g.uniform(0.8, 1.0, n), g.uniform(0.3, 0.4, n), g.normal(size=(n, 3)), g.normal(size=(n, 3)))]
    d = [v.double() for v in t]
    dbox = torch.tensor(box, device="cuda").float().double() if pbc else None
    ref, edge = _fp64(d[0], d[1], d[2], d[3], dbox)
    refp, _ = _fp64(d[0], d[1], d[2], d[4], dbox)
    out = [t[4], t[3]] if inplace else [torch.full((n, 3), float("nan"), device="cuda") for _ in range(2)]
    rc = lib.t9gb_ufield_noalloc(n, (C.c_double * 3)(*box) if pbc else None, CUTOFF,
                                 *[C.c_void_p(v.data_ptr()) for v in t + out],
                                 C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == gpu_lib.T9GB_OK
    torch.cuda.synchronize()
    for o, r in ((out[0], ref), (out[1], refp)):
        o, r = o.double()[~edge], r[~edge]
        assert torch.isfinite(o).all()
        assert (o - r).norm() <= FIELD_RTOL * r.norm()
