"""The calls that a user of this library makes, as cases to be timed and compared.

Each case is one kind of call on one box.  Boxes are the seeded AMOEBA water boxes of
tinker-gpu_gb300/systems.py (its named configurations, and boxes between them at the same
density, with vacancies, ions and the PME grid that Tinker's rule of 1.2 points per A gives).

  noalloc   t9gb_ufield_noalloc: the mutual field for callers that may not allocate
  induce    one dipole solve: alpha E start, ASPC / Gear ring, learned extrapolation or the
            trained network's start; coordinates on the device, or on the host through t9gb_induce_host
  cluster   the same without periodic box or Ewald sum (gas-phase droplet)
  fields    dfield, ufield and the sparse preconditioner as separate calls, as a host program
            with a solver of its own makes them
  energy    a single point: multipole + polarization energy, gradient and virial, van der Waals
            and valence energy and gradient
  md        velocity-Verlet steps of the whole water force field under the Bussi thermostat

Solves run over frames of a librating trajectory with a period of 240 fs, so that a state can be
used for any number of passes and the predictor's ring always sees smooth motion.
"""
import ctypes as C
import dataclasses
import functools
import importlib
import math

import numpy as np
import torch

abi = importlib.import_module("tinker-gpu_gb300.abi")
systems = importlib.import_module("tinker-gpu_gb300.systems")
units = importlib.import_module("tinker-gpu_gb300.units")

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"
PERIOD = 240  # frames (fs) of the periodic trajectory
HISTORY = 20  # solves before the first pass: the ASPC ring holds 16 frames, the fit starts at 2
KELVIN = 298.0
MASS = {systems.WATER_O: 15.999, systems.WATER_H: 1.008, systems.NA_ION: 22.99, systems.CL_ION: 35.453}
PREDICTORS = {"none": 0, "aspc": 1, "gear": 2}

BOXES = {name: dict(nside=c["nside"], box=c["box"], nfft=c["nfft"], sites=c.get("n_sites", c["nside"] ** 3),
                    ion_pairs=c.get("n_ion_pairs", 0)) for name, c in systems.CONFIGS.items()}


def listed():
    small, mid, salt, large = (BOXES[k] for k in ("water648", "water12288", "nacl23142", "water98304"))
    return [
        # a real-time loop that asks for the field of a small solvent box: one launch-bound call
        dict(name="noalloc-648", kind="noalloc", **small, cutoff=7.0),
        # one geometry, no history: what an ANALYZE run or an optimiser's first step pays, PME 24^3
        dict(name="induce-648", kind="induce", **small, predictor="none"),
        # molecular dynamics of a small box: every launch counts
        dict(name="md-648", kind="md", **small, predictor="aspc", steps=10),
        # a gas-phase droplet: no box, no Ewald sum, all pairs
        dict(name="cluster-1500", kind="cluster", nside=8, box=24.64, nfft=32, sites=500, ion_pairs=0, predictor="none"),
        # the fields and the preconditioner on their own, on the box of the headline benchmark
        dict(name="fields-12288", kind="fields", **mid),
        # the headline benchmark: a solve with the ASPC ring full, PME 64^3
        dict(name="induce-12288", kind="induce", **mid, predictor="aspc"),
        # the same end to end from host memory, with the learned extrapolation of the ring
        dict(name="induce-host-12288", kind="induce", **mid, predictor="aspc", extrapolation=8, host=True),
        # online training of the network and solves that start from it
        dict(name="learn-12288", kind="induce", **mid, predictor="none", learn=True),
        # a single point of a salt solution with vacancies: 23,142 atoms, PME 72^3 (ragged sizes), virial
        dict(name="energy-23142", kind="energy", **salt),
        # molecular dynamics of the headline box
        dict(name="md-12288", kind="md", **mid, predictor="aspc", steps=10),
        # the largest benchmark box: one solve, PME 128^3
        dict(name="induce-98304", kind="induce", **large, predictor="aspc"),
        # molecular dynamics of the largest box, with the learned extrapolation
        dict(name="md-98304", kind="md", **large, predictor="aspc", extrapolation=8, steps=5),
    ]


def _grid(box):
    """Smallest even PME grid of factors 2, 3 and 5 with 1.2 points per A (Tinker's default)."""
    n = max(16, int(math.ceil(1.2 * box)))
    while True:
        m = n
        for f in (2, 3, 5):
            while m % f == 0:
                m //= f
        if m == 1 and n % 2 == 0:
            return n
        n += 1


def _draw_box(rng, lo, hi):
    """A cubic water box of lo..hi molecules at the density of the named configurations."""
    m = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    nside = max(6, int(math.ceil(m ** (1 / 3))))
    sites = min(nside ** 3, max(m, int(0.93 * nside ** 3)))
    box = round(rng.uniform(3.08, 3.107) * nside, 3)
    return dict(nside=nside, box=box, nfft=_grid(box), sites=sites,
                ion_pairs=rng.choice([0, 0, sites // 370]) if sites > 370 else 0)


def draw(rng):
    kind = rng.choice(["noalloc", "induce", "induce", "induce", "cluster", "fields", "energy", "md", "md"])
    if kind == "noalloc":  # up to the entry point's 8,192 atoms
        b = _draw_box(rng, 216, 2500)
        return dict(kind=kind, **b, cutoff=round(rng.uniform(6.0, 9.0), 2))
    if kind == "cluster":
        b = _draw_box(rng, 60, 700)
        b["sites"] = min(b["sites"], int(math.exp(rng.uniform(math.log(40), math.log(700)))))
        return dict(kind=kind, **dict(b, ion_pairs=0), predictor="none")
    b = _draw_box(rng, 216, 29000)
    if kind == "induce":
        p = rng.choice(["none", "aspc", "aspc", "gear"])
        c = dict(kind=kind, **b, predictor=p, host=rng.random() < 0.3)
        if p != "none" and rng.random() < 0.5:
            c["extrapolation"] = 5 if p == "gear" else rng.choice([6, 8])
        if p == "none" and not c["host"] and rng.random() < 0.3:
            c["learn"] = True
        return c
    if kind == "md":
        c = dict(kind=kind, **b, predictor="aspc", steps=rng.choice([1, 2, 4]))
        if rng.random() < 0.5:
            c["extrapolation"] = 8
        return c
    return dict(kind=kind, **b)


# ---------------------------------------------------------------------------
# state


@functools.lru_cache(maxsize=None)
def _topology(kind, nside, box, nfft, sites, ion_pairs):
    """Topology and force field (the program's parameter files); positions come from the seed."""
    full = kind in ("energy", "md")
    s = systems.make_config("water648", vdw=full, valence=full, nside=nside, box=box, seed=5, nfft=nfft, n_sites=sites,
                            n_ion_pairs=ion_pairs)
    if kind == "cluster":
        lat = s.lattice
        s = dataclasses.replace(s, box=None, settings=dict(s.settings, use_ewald=0, ewald_cutoff=1.0e9, nfft=(0, 0, 0),
                                                           aewald=0.0))
        s.lattice = lat
    return s


def _system(case):
    return _topology(case["kind"], case["nside"], case["box"], case["nfft"], case["sites"], case["ion_pairs"])


def _frames(s, seed, count, stride=1):
    """Frames [count][n][3] (float64, on the GPU) of the molecules' periodic motion about their
    sites: translation by up to 0.15 A (80-120 fs), libration by up to 20 degrees (40-120 fs)."""
    g = torch.Generator().manual_seed(1000003 * seed + 17)
    m = len(s.lattice.centers)

    def unit():
        d = torch.randn(m, 3, generator=g, dtype=torch.float64)
        return d / d.norm(dim=1, keepdim=True)

    td, ra = 0.15 * unit(), unit()
    # whole turns in a period: 2-3 of the translation, 2-6 of the libration
    tw, rw = (2 * math.pi / PERIOD * torch.randint(2, top, (m,), generator=g).double() for top in (4, 7))
    tp, rp = (2 * math.pi * torch.rand(m, generator=g, dtype=torch.float64) for _ in range(2))
    td, ra, tw, rw, tp, rp = (v.to(DEVICE) for v in (td, ra, tw, rw, tp, rp))
    c0, rot = (torch.as_tensor(v, device=DEVICE) for v in (s.lattice.centers, s.lattice.rot))
    # atom -> molecule, and the body-frame site: water's O, H, H or an ion at the centre
    size = torch.as_tensor(s.mol_size, device=DEVICE)
    mol = torch.repeat_interleave(torch.arange(m, device=DEVICE), size)
    at = torch.arange(s.n, device=DEVICE) - torch.as_tensor(s.mol_start, device=DEVICE)[mol]
    body = torch.as_tensor(systems.water_geometry(), device=DEVICE)[at]
    arm = torch.einsum("nij,nj->ni", rot[mol], body)
    k = ra[mol]
    out = torch.empty((count, s.n, 3), dtype=torch.float64, device=DEVICE)
    for f in range(count):
        t = stride * f
        a = (math.radians(20.0) * torch.sin(rw * t + rp))[mol][:, None]
        turned = arm * torch.cos(a) + torch.linalg.cross(k, arm) * torch.sin(a) + k * (k * arm).sum(1, keepdim=True) * (1 - torch.cos(a))
        out[f] = (c0 + td * torch.sin(tw * t + tp)[:, None])[mol] + turned
    return out


def _dipoles(n, seed):
    g = torch.Generator(device=DEVICE).manual_seed(seed + 5)
    return [0.05 * torch.randn(n, 3, generator=g, device=DEVICE) for _ in range(2)]


def _masses(s):
    return np.array([MASS[int(t)] for t in s.types])


def _solve(st):
    """One solve on the next frame, as an MD driver with forces of its own does it."""
    e, f = st["engine"], st["frames"][st["next"] % len(st["frames"])]
    st["next"] += 1
    if st["host"]:
        return e.induce_host(f, *st["out"])
    e.set_xyz_device(f)
    e.mpole_init()
    return e.induce(st["out"])


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def prepare(case, seed):
    s = _system(case)
    n, kind = s.n, case["kind"]
    stream = torch.cuda.Stream()
    trajectory = case.get("predictor", "none") != "none" or bool(case.get("learn"))
    if kind == "md":
        x = _frames(s, seed, 1)[0].cpu().numpy()
    else:
        fr = _frames(s, seed, PERIOD if trajectory else 8, 1 if trajectory else PERIOD // 8)
        host = bool(case.get("host"))
        fr = list(fr.cpu().numpy()) if host else fr.float()
        x = np.asarray(fr[0], dtype=np.float64) if host else fr[0].double().cpu().numpy()
    torch.cuda.synchronize()
    if kind == "noalloc":
        f32 = dict(dtype=torch.float32, device=DEVICE)
        return dict(kind=kind, n=n, lib=abi.load(), box=(C.c_double * 3)(*s.box), cutoff=case["cutoff"], stream=stream,
                    ins=[fr[0].contiguous(), torch.tensor(s.pdamp, **f32), torch.tensor(s.thole, **f32)] + _dipoles(n, seed),
                    out=[torch.zeros(n, 3, **f32) for _ in range(2)])
    e = abi.Engine(s, predictor=PREDICTORS[case.get("predictor", "none")], stream=stream)
    e.prepare(x)
    if case.get("extrapolation"):
        e.learn_extrapolation(case["extrapolation"])
    st = dict(kind=kind, n=n, engine=e, stream=stream)
    if kind == "md":
        mass = _masses(s)
        v = np.random.default_rng(seed).normal(size=(n, 3)) * np.sqrt(1.987204259e-3 * KELVIN * 418.4 / mass)[:, None]
        e.md_init(x, mass, v)
        # the thermostat takes up the heat of the random orientations; the predictor's ring fills
        e.md_run(30, 0.001, thermostat=1, kelvin=KELVIN, tau_ps=0.01, seed=seed)
        st.update(steps=case["steps"], seed=seed, out=torch.zeros(n, 3, device=DEVICE))
        return st
    st.update(frames=fr, next=0, host=host, learn=bool(case.get("learn")))
    if kind == "fields":
        st.update(dip=_dipoles(n, seed), out=[torch.zeros(n, 3, device=DEVICE) for _ in range(6)])
    elif kind in ("induce", "cluster"):
        st["out"] = [np.zeros((n, 3)) for _ in range(2)] if host else [torch.zeros(n, 3, device=DEVICE) for _ in range(2)]
        if st["learn"]:
            e.learn_reset(seed=1 + seed % 1000)
            e.learn_config(abi.LEARN_TRAIN | abi.LEARN_USE)
            e.learn_policy(16)
        if trajectory:
            for _ in range(HISTORY):
                _solve(st)
    torch.cuda.synchronize()
    return st


def _f32(v):
    """Energies, virials and host dipoles are FP32 results in FP64 words."""
    return torch.as_tensor(np.asarray(v, dtype=np.float32))


def run(st):
    kind = st["kind"]
    if kind == "noalloc":
        rc = st["lib"].t9gb_ufield_noalloc(st["n"], st["box"], st["cutoff"], *[_ptr(t) for t in st["ins"] + st["out"]],
                                           C.c_void_p(st["stream"].cuda_stream))
        if rc:
            raise RuntimeError("t9gb_ufield_noalloc: status %d" % rc)
        return st["out"]
    e = st["engine"]
    with torch.cuda.stream(st["stream"]):
        if kind == "md":
            _, _, rc = e.md_run(st["steps"], 0.001, thermostat=1, kelvin=KELVIN, tau_ps=0.1, seed=st["seed"])
            if rc:
                raise RuntimeError("md_run: status %d" % rc)
            # a saved frame: positions, velocities and induced dipoles (the FP64 trajectory at the
            # precision of its FP32 forces)
            e.md_positions_device(st["out"])
            _, v, _ = e.md_state()
            return [st["out"], _f32(v), *e.uind()]
        if kind == "fields":
            f = st["frames"][st["next"] % len(st["frames"])]
            st["next"] += 1
            e.set_xyz_device(f)
            e.mpole_init()
            o, d = [_ptr(t) for t in st["out"]], [_ptr(t) for t in st["dip"]]
            for rc in (e.lib.t9gb_dfield(e.h, o[0], o[1]), e.lib.t9gb_ufield(e.h, *d, o[2], o[3]),
                       e.lib.t9gb_sparse_precond_apply(e.h, *d, o[4], o[5])):
                if rc:
                    raise RuntimeError("fields: status %d" % rc)
            return st["out"]
        if kind == "energy":
            f = st["frames"][st["next"] % len(st["frames"])]
            st["next"] += 1
            e.set_xyz_device(f)
            e.mpole_init()
            _, g, vir = e.emplar(abi.CALC_ENERGY | abi.CALC_GRAD | abi.CALC_VIRIAL)
            parts = e.energy_components()
            eh, gh = e.ehal()
            ev, gv = e.evalence()
            return dict(grad=g, virial=_f32(vir), parts=_f32(parts), hal=_f32([eh]), grad_hal=gh, valence=_f32([ev]),
                        grad_valence=gv)
        ud, up, rc = _solve(st)
        if rc:
            raise RuntimeError("induce: status %d" % rc)
        if st["host"]:
            ud, up = _f32(ud), _f32(up)
        return [ud, up, _f32(e.learn_weights())] if st["learn"] else [ud, up]


# ---------------------------------------------------------------------------
# work


def work(case):
    """Inputs read once, outputs written once, and the arithmetic of the fewest passes: pair terms
    within the cutoffs (each pair once), B-spline points, real-to-complex transforms."""
    s = _system(case)
    n = s.n
    density = n / case["box"] ** 3
    per = lambda rc: n * density * 4 / 3 * math.pi * rc ** 3 / 2  # noqa: E731
    pairs, near = per(7.0), per(6.5)
    if case["kind"] == "cluster":
        pairs = n * (n - 1) / 2
        near = min(pairs, near)
    points = 0 if case["kind"] == "cluster" else case["nfft"] ** 3
    fft = 2 * 2.5 * points * math.log2(points) if points else 0  # forward and back, one real grid
    recip = lambda grids: grids * (n * 125 * 12 + fft) if points else 0  # noqa: E731
    atom_in = 12 + 40 + 12 + 16 + 36  # coordinates, multipoles, polarizability and damping, frame, exclusions
    dfield = pairs * 130 + recip(1)
    ufield = pairs * 70 + recip(2)
    precond = near * 50
    # the PCG's fewest iterations are three, and the starting residual needs one more field
    solve = dfield + 4 * (ufield + precond)
    hal = n * density * 4 / 3 * math.pi * 9.0 ** 3 / 2 * 40
    forces = pairs * 700 + recip(3)
    if case["kind"] == "noalloc":
        return dict(bytes=n * (12 + 8 + 24 + 24), flops=per(case["cutoff"]) * 70)
    if case["kind"] == "fields":
        return dict(bytes=n * (atom_in + 24 + 72), flops=dfield + ufield + precond)
    if case["kind"] == "energy":
        return dict(bytes=n * (atom_in + 24 + 36), flops=solve + forces + hal)
    if case["kind"] == "md":  # positions and velocities are FP64
        return dict(bytes=case["steps"] * n * (atom_in + 24 + 2 * 48), flops=case["steps"] * (solve + forces + hal))
    ring = {"none": 0, "aspc": 16, "gear": 6}[case["predictor"]]
    net = 3 * 2 * 2 * n * (32 * 64 + 64 * 64 + 64 * 3) if case.get("learn") else 0
    return dict(bytes=n * (atom_in + 24 + 24 * ring), flops=solve + net)


# ---------------------------------------------------------------------------
# the same quantities in 64 bits, from the published equations (Thole-damped AMOEBA multipoles,
# smooth PME of order 5), with torch's FFT and autograd


def _image(d, box):
    return d if box is None else d - box * torch.round(d / box)


def _unit(v):
    return v / v.norm(dim=1, keepdim=True)


class _Exact:
    def __init__(self, s, x):
        self.s, self.n = s, s.n
        f = lambda v: torch.as_tensor(np.array(v, dtype=np.float64), device=DEVICE)  # noqa: E731
        self.x = x.double().to(DEVICE)
        self.box = None if s.box is None else f(s.box)
        self.alpha, self.thole, self.pdamp, self.pole = f(s.polarity), f(s.thole), f(s.pdamp), f(s.pole)
        self.ewald = bool(s.settings["use_ewald"])
        self.aew = s.settings["aewald"]
        self.frames = torch.as_tensor(np.array(s.frames), device=DEVICE).long()
        ik = torch.as_tensor(np.array(s.excl_ik), device=DEVICE).long().reshape(-1, 2)
        self.ekey, o = (ik[:, 0] * s.n + ik[:, 1]).sort()
        self.escale = f(s.excl_scale).reshape(-1, 4)[o]
        self.eps = torch.zeros(3, 3, dtype=torch.float64, device=DEVICE)  # strain of box and coordinates
        if self.ewald:
            self.nf = [int(k) for k in s.settings["nfft"]]
            self._influence()

    def pairs(self, x, cut):
        """i < k within the cutoff, by images of the unstrained box."""
        step, out = max(1, 60_000_000 // self.n), []
        for a in range(0, self.n, step):
            d = _image(x[None, :, :] - x[a:a + step, None, :], self.box)
            hit = ((d * d).sum(2) <= cut * cut).nonzero()
            hit[:, 0] += a
            out.append(hit[hit[:, 0] < hit[:, 1]])
        p = torch.cat(out)
        return p[:, 0], p[:, 1]

    def scales(self, i, k):
        key = i * self.n + k
        sc = torch.ones(len(key), 4, dtype=torch.float64, device=DEVICE)
        if len(self.ekey):
            at = torch.searchsorted(self.ekey, key).clamp(max=len(self.ekey) - 1)
            hit = self.ekey[at] == key
            sc[hit] = self.escale[at[hit]]
        return sc

    def strained(self, v):
        return v + v @ self.eps.T

    def separation(self, x, i, k):
        return self.strained(_image(x[k] - x[i], self.box))

    def rotate(self, x):
        """Charge [n], dipole [n][3] and quadrupole [n][3][3] in the global frame."""
        kind = self.frames[:, 3]
        rows = torch.zeros(self.n, 3, 3, dtype=torch.float64, device=DEVICE) + torch.eye(3, dtype=torch.float64, device=DEVICE)
        w = (kind > 0).nonzero()[:, 0]
        i, bis = w, (kind[w] == 3)[:, None]
        z = _unit(self.separation(x, i, self.frames[w, 0]))
        a = _unit(self.separation(x, i, self.frames[w, 1]))
        z = torch.where(bis, _unit(z + a), z)
        a = _unit(a - (a * z).sum(1, keepdim=True) * z)
        rows = rows.index_put((w,), torch.stack([a, torch.linalg.cross(z, a), z], 1))
        p = self.pole
        q = torch.stack([p[:, [4, 7, 8]], p[:, [7, 5, 9]], p[:, [8, 9, 6]]], 1)
        return p[:, 0], torch.einsum("nj,njc->nc", p[:, 1:4], rows), torch.einsum("njk,nja,nkb->nab", q, rows, rows)

    def bn(self, r, order):
        """B_0..B_order of erfc(a r)/r, or of 1/r without the Ewald sum."""
        if not self.ewald:
            b = [1 / r]
            for j in range(1, order + 1):
                b.append((2 * j - 1) * b[-1] / (r * r))
            return b
        b, pre = [torch.erfc(self.aew * r) / r], 1 / (math.sqrt(math.pi) * self.aew)
        ex = torch.exp(-(self.aew * r) ** 2)
        for j in range(1, order + 1):
            pre *= 2 * self.aew ** 2
            b.append(((2 * j - 1) * b[-1] + pre * ex) / (r * r))
        return b

    def damped(self, r, i, k, sc, order):
        """B_1..B_order with Thole damping and the pair's scale."""
        pd = self.pdamp[i] * self.pdamp[k]
        a = torch.minimum(self.thole[i], self.thole[k]) * (r / pd) ** 3
        ex = torch.exp(-a)
        lam = [1 - ex, 1 - ex * (1 + a), 1 - ex * (1 + a + 0.6 * a * a)]
        b, rr, out = self.bn(r, order), 1 / r, []
        for j in range(1, order + 1):
            rr = rr * (2 * j - 1) / (r * r)
            out.append(b[j] - (1 - sc * lam[j - 1]) * rr if self.ewald else sc * lam[j - 1] * rr)
        return out

    def perm_fields(self, x, pair, M):
        """Real-space part of the d- and p-scaled permanent fields [n][2][3]."""
        i, k = pair
        d = self.separation(x, i, k)
        r = d.norm(dim=1)
        q, mu, th = M
        tk, ti = torch.einsum("pab,pb->pa", th[k], d), torch.einsum("pab,pb->pa", th[i], d)
        dk, di = (mu[k] * d).sum(1), (mu[i] * d).sum(1)
        qk, qi = (tk * d).sum(1), (ti * d).sum(1)
        sc, out = self.scales(i, k), []
        for col in (1, 2):
            b1, b2, b3 = (v[:, None] for v in self.damped(r, i, k, sc[:, col], 3))
            fi = -(b1 * q[k][:, None] - b2 * dk[:, None] + b3 * qk[:, None]) * d - b1 * mu[k] + 2 * b2 * tk
            fk = (b1 * q[i][:, None] + b2 * di[:, None] + b3 * qi[:, None]) * d - b1 * mu[i] - 2 * b2 * ti
            out.append(torch.zeros_like(x).index_add(0, i, fi).index_add(0, k, fk))
        return torch.stack(out, 1)

    def tensor(self, x, pair, damp=True):
        """Distance vector and the two radial factors of the mutual dipole field."""
        i, k = pair
        d = self.separation(x, i, k)
        b1, b2 = self.damped(d.norm(dim=1), i, k, self.scales(i, k)[:, 3], 2)
        return d, b1, b2

    def mutual(self, t, pair, u):
        """Real-space mutual field of u [n][m][3]."""
        (d, b1, b2), (i, k) = t, pair
        d, b1, b2 = d[:, None, :], b1[:, None, None], b2[:, None, None]
        f = lambda v: b2 * (v * d).sum(2, keepdim=True) * d - b1 * v  # noqa: E731
        return torch.zeros_like(u).index_add(0, i, f(u[k])).index_add(0, k, f(u[i]))

    # smooth PME
    def _influence(self):
        mod = []
        for n in self.nf:
            m = np.array([1 / 24, 11 / 24, 11 / 24, 1 / 24])  # M5 at the integers 1..4
            kk = np.arange(n)
            b = np.abs((m[None, :] * np.exp(2j * math.pi * kk[:, None] * np.arange(4)[None, :] / n)).sum(1)) ** 2
            for j in range(1, n - 1):
                if b[j] < 1e-7:
                    b[j] = 0.5 * (b[j - 1] + b[j + 1])
            # optimal zeta of the Euler spline
            z = np.where(kk + 1 > n // 2, kk - n, kk).astype(float)
            s1, s2 = np.ones(n), np.ones(n)
            with np.errstate(invalid="ignore", divide="ignore"):
                for j in range(1, 51):
                    for g in (z / (z + n * j), z / (z - n * j)):
                        s1 += g ** 5
                        s2 += g ** 10
            mod.append(torch.as_tensor(b * (s2 / s1) ** 2, device=DEVICE))
        self.mod = mod

    def green(self, Hinv):
        """Influence function on the reciprocal grid of the (strained) cell."""
        k = [torch.as_tensor(np.where(np.arange(n) < (n + 1) // 2, np.arange(n), np.arange(n) - n), device=DEVICE).double() for n in self.nf]
        k1, k2, k3 = k[0][:, None, None], k[1][None, :, None], k[2][None, None, :self.nf[2] // 2 + 1].abs()
        hsq = sum((k1 * Hinv[0, a] + k2 * Hinv[1, a] + k3 * Hinv[2, a]) ** 2 for a in range(3))
        zero = torch.zeros_like(hsq, dtype=torch.bool)
        zero[0, 0, 0] = True
        hsq = torch.where(zero, torch.ones_like(hsq), hsq)
        term = -(math.pi / self.aew) ** 2 * hsq
        vol = 1 / torch.linalg.det(Hinv)
        b = self.mod[0][:, None, None] * self.mod[1][None, :, None] * self.mod[2][None, None, :self.nf[2] // 2 + 1]
        g = torch.exp(term) / (hsq * math.pi * vol * b)
        return torch.where(zero | (term <= -50), torch.zeros_like(g), g)

    def sites(self, x):
        """Grid indices [n][125] and the spline values and first two derivatives by axis."""
        th, at = [], []
        for a in range(3):
            w = x[:, a] / self.box[a] + 0.5
            w = self.nf[a] * (w - torch.floor(w.detach()))
            g = torch.floor(w.detach())
            w = w - g
            m = {2: torch.stack([1 - w, w], 1)}
            for o in range(3, 6):
                lo = torch.nn.functional.pad(m[o - 1], (1, 1))
                j = torch.arange(1, o + 1, device=DEVICE)[None, :]
                m[o] = ((w[:, None] + o - j) * lo[:, :-1] + (j - w[:, None]) * lo[:, 1:]) / (o - 1)
            d = lambda v: -torch.diff(torch.nn.functional.pad(v, (1, 1)), dim=1)  # noqa: E731
            th.append([m[5], d(m[4]), d(d(m[3]))])
            at.append((g.long()[:, None] - 4 + torch.arange(5, device=DEVICE)[None, :]) % self.nf[a])
        idx = ((at[0][:, :, None, None] * self.nf[1] + at[1][:, None, :, None]) * self.nf[2] + at[2][:, None, None, :]).reshape(self.n, -1)
        return idx, th

    def cell(self):
        Hinv = torch.diag(1 / self.box) @ torch.linalg.inv(torch.eye(3, dtype=torch.float64, device=DEVICE) + self.eps)
        return Hinv, torch.diag(torch.tensor(self.nf, dtype=torch.float64, device=DEVICE)) @ Hinv

    def spread(self, site, T, q=None, mu=None, quad=None):
        idx, (X, Y, Z) = site
        prod = lambda a, b, c, v: torch.einsum("ni,nj,nk,n->nijk", X[a], Y[b], Z[c], v)  # noqa: E731
        val = 0
        if q is not None:
            val = val + prod(0, 0, 0, q)
        if mu is not None:
            f = mu @ T.T
            val = val + prod(1, 0, 0, f[:, 0]) + prod(0, 1, 0, f[:, 1]) + prod(0, 0, 1, f[:, 2])
        if quad is not None:
            f = torch.einsum("fa,nab,gb->nfg", T, quad, T)
            val = val + prod(2, 0, 0, f[:, 0, 0]) + prod(0, 2, 0, f[:, 1, 1]) + prod(0, 0, 2, f[:, 2, 2]) + \
                2 * (prod(1, 1, 0, f[:, 0, 1]) + prod(1, 0, 1, f[:, 0, 2]) + prod(0, 1, 1, f[:, 1, 2]))
        grid = torch.zeros(self.nf[0] * self.nf[1] * self.nf[2], dtype=torch.float64, device=DEVICE)
        return grid.index_add(0, idx.reshape(-1), val.reshape(-1))

    def potential(self, grid, G):
        n = self.nf[0] * self.nf[1] * self.nf[2]
        return n * torch.fft.irfftn(torch.fft.rfftn(grid.reshape(self.nf)) * G, s=self.nf).reshape(-1)

    def grid_field(self, phi, site, T):
        idx, (X, Y, Z) = site
        p = phi[idx].reshape(self.n, 5, 5, 5)
        g = torch.stack([torch.einsum("nijk,ni,nj,nk->n", p, X[a], Y[b], Z[c]) for a, b, c in ((1, 0, 0), (0, 1, 0), (0, 0, 1))], 1)
        return -(g @ T)

    def setup(self):
        self.pair = self.pairs(self.x, min(self.s.settings["ewald_cutoff"], 1e6))
        self.M = self.rotate(self.x)
        self.t = self.tensor(self.x, self.pair)
        if self.ewald:
            Hinv, self.T = self.cell()
            self.G, self.site = self.green(Hinv), self.sites(self.x)
            self.self_term = 4 * self.aew ** 3 / (3 * math.sqrt(math.pi))
        return self

    def dfield(self):
        f = self.perm_fields(self.x, self.pair, self.M)
        if self.ewald:
            phi = self.potential(self.spread(self.site, self.T, *self.M), self.G)
            f = f + (self.grid_field(phi, self.site, self.T) + self.self_term * self.M[1])[:, None, :]
        return f

    def ufield(self, u):
        f = self.mutual(self.t, self.pair, u)
        if self.ewald:
            rec = [self.grid_field(self.potential(self.spread(self.site, self.T, mu=u[:, c]), self.G), self.site, self.T) for c in range(u.shape[1])]
            f = f + torch.stack(rec, 1) + self.self_term * u
        return f

    def precond(self, r):
        s = self.s.settings
        pair = self.pairs(self.x, s["usolve_cutoff"] + s["pbuffer"])
        i, k = pair
        was, self.ewald = self.ewald, False  # the preconditioner's tensor is Thole-damped without the Ewald sum
        d, b1, b2 = self.tensor(self.x, pair)
        self.ewald = was
        ak = self.alpha[i] * self.alpha[k]
        return s["udiag"] * self.alpha[:, None, None] * r + self.mutual((d, ak * b1, ak * b2), pair, r)

    def induce(self):
        """Dipoles [n][2][3] to a residual of 1e-11 D, by conjugate gradients with alpha as preconditioner."""
        a = self.alpha[:, None, None]
        dot = lambda u, v: (u * v).sum((0, 2), keepdim=True)  # noqa: E731
        u = a * self.dfield()
        r = self.ufield(u)
        z = a * r
        p, rz = z, dot(r, z)
        for _ in range(200):
            v = p / a - self.ufield(p)
            step = rz / dot(p, v)
            u, r = u + step * p, r - step * v
            if float((dot(r, r) / self.n).sqrt().max()) * units.DEBYE < 1e-11:
                break
            z = a * r
            new = dot(r, z)
            p, rz = z + new / rz * p, new
        return u

    def forces(self, u):
        """Gradient and virial of multipole + polarization energy at dipoles u, and [real, recip, self, polar]."""
        f = units.ELECTRIC
        x, self.eps = self.x.clone().requires_grad_(), self.eps.clone().requires_grad_()
        ud, up = u[:, 0], u[:, 1]
        i, k = self.pair
        M = q, mu, th = self.rotate(x)
        d = self.separation(x, i, k)
        r = d.norm(dim=1)
        tk, ti = torch.einsum("pab,pb->pa", th[k], d), torch.einsum("pab,pb->pa", th[i], d)
        dk, di, qk, qi = ((v * d).sum(1) for v in (mu[k], mu[i], tk, ti))
        terms = [q[i] * q[k], q[k] * di - q[i] * dk + (mu[i] * mu[k]).sum(1),
                 q[i] * qk + q[k] * qi - di * dk + 2 * ((mu[k] * ti).sum(1) - (mu[i] * tk).sum(1) + (th[i] * th[k]).sum((1, 2))),
                 di * qk - dk * qi - 4 * (ti * tk).sum(1), qi * qk]
        b, m = self.bn(r, 4), self.scales(i, k)[:, 0]
        rr, e_real = 1 / r, 0
        for j in range(5):
            rr = rr if j == 0 else rr * (2 * j - 1) / (r * r)
            e_real = e_real + (terms[j] * (b[j] + (m - 1) * rr if self.ewald else m * rr)).sum()
        e_real = f * e_real
        E = self.perm_fields(x, self.pair, M)
        t = self.tensor(x, self.pair)
        g_pol = (up * E[:, 0]).sum() + (ud * E[:, 1]).sum() + (ud * self.mutual(t, self.pair, up[:, None])[:, 0]).sum()
        e_recip = e_self = torch.zeros((), dtype=torch.float64, device=DEVICE)
        if self.ewald:
            Hinv, T = self.cell()
            G, site = self.green(Hinv), self.sites(x)
            gm, gd, gp = self.spread(site, T, q, mu, th), self.spread(site, T, mu=ud), self.spread(site, T, mu=up)
            pm = self.potential(gm, G)
            e_recip = 0.5 * f * (gm * pm).sum()
            a = self.aew
            e_self = -f * a / math.sqrt(math.pi) * (q * q + 2 * a * a * ((mu * mu).sum(1) / 3 + 0.8 * a * a * (th * th).sum((1, 2)))).sum()
            g_pol = g_pol - ((gp + gd) * pm).sum() - (gd * self.potential(gp, G)).sum() + \
                self.self_term * ((up * mu).sum() + (ud * mu).sum() + (ud * up).sum())
        total = e_real + e_recip + e_self - 0.5 * f * g_pol
        grad, vir = torch.autograd.grad(total, (x, self.eps))
        self.eps = self.eps.detach() * 0
        e_pol = -0.5 * f * (ud * self.dfield()[:, 1]).sum()
        return grad, 0.5 * (vir + vir.T), torch.stack([e_real, e_recip, e_self, e_pol]).detach()

    def hal(self):
        """Buffered 14-7 energy and gradient (reduced hydrogen sites, fifth-order taper)."""
        v = self.s.vdw
        f = lambda a: torch.as_tensor(np.array(a), device=DEVICE)  # noqa: E731
        x = self.x.clone().requires_grad_()
        par = f(v.parent).long()
        sx = x[par] + f(v.red)[:, None] * _image(x - x[par], self.box)
        i, k = self.pairs(sx.detach(), v.off)
        key, order = (f(v.scaled_ik).long()[:, 0] * self.n + f(v.scaled_ik).long()[:, 1]).sort()
        at = torch.searchsorted(key, i * self.n + k).clamp(max=len(key) - 1)
        w = torch.where(key[at] == i * self.n + k, f(v.scaled_v)[order][at], torch.ones_like(self.x[i, 0]))
        r = _image(sx[k] - sx[i], self.box).norm(dim=1)
        ty = f(v.vtype).long()
        rho = r / f(v.radmin)[ty[i], ty[k]]
        e = w * f(v.epsilon)[ty[i], ty[k]] * (1.07 / (rho + 0.07)) ** 7 * (1.12 / (rho ** 7 + 0.12) - 2)
        y = (r - v.off) / (v.taper - v.off)
        e = torch.where(r > v.taper, e * y ** 3 * (6 * y * y - 15 * y + 10), e).sum()
        return e.detach().reshape(1), torch.autograd.grad(e, x)[0]

    def valence(self):
        v = self.s.valence
        f = lambda a, w: torch.as_tensor(np.array(a, dtype=np.float64), device=DEVICE).reshape(-1, w)  # noqa: E731
        x = self.x.clone().requires_grad_()
        vec = lambda a, b: _image(x[a.long()] - x[b.long()], self.box)  # noqa: E731
        b, a, u = f(v.bonds, 4), f(v.angles, 5), f(v.ureys, 5)
        t = vec(b[:, 0], b[:, 1]).norm(dim=1) - b[:, 3]
        e = (b[:, 2] * t * t * (1 + v.bond_cubic * t + v.bond_quartic * t * t)).sum()
        p, q = vec(a[:, 0], a[:, 1]), vec(a[:, 2], a[:, 1])
        t = torch.rad2deg(torch.arccos((p * q).sum(1) / (p.norm(dim=1) * q.norm(dim=1)))) - a[:, 4]
        c = v.angle_terms
        e = e + ((math.pi / 180) ** 2 * a[:, 3] * t ** 2 * (1 + c[0] * t + c[1] * t ** 2 + c[2] * t ** 3 + c[3] * t ** 4)).sum()
        t = vec(u[:, 0], u[:, 2]).norm(dim=1) - u[:, 4]
        e = e + (u[:, 3] * t * t * (1 + v.urey_cubic * t + v.urey_quartic * t * t)).sum()
        return e.detach().reshape(1), torch.autograd.grad(e, x)[0]


def exact(case, seed):
    """The first pass's outputs in 64 bits.  A trajectory has no such value (None): its steps
    amplify any rounding, and what they are made of is in the other cases."""
    kind = case["kind"]
    if kind == "md":
        return None
    s = _system(case)
    if kind == "noalloc":
        x = _frames(s, seed, 1)[0].float()
        one = dataclasses.replace(s, excl_ik=np.zeros((0, 2), dtype=np.int32), excl_scale=np.zeros((0, 4)),
                                  settings=dict(s.settings, use_ewald=0))
        e = _Exact(one, x)
        pair = e.pairs(e.x, case["cutoff"])
        f = e.mutual(e.tensor(e.x, pair), pair, torch.stack([d.double() for d in _dipoles(s.n, seed)], 1))
        return [f[:, 0], f[:, 1]]
    ring = case.get("predictor", "none") != "none" or bool(case.get("learn"))
    x = _frames(s, seed, HISTORY + 1 if ring else 1)[-1]
    e = _Exact(s, x if case.get("host") else x.float()).setup()
    if kind == "fields":
        d = torch.stack([v.double() for v in _dipoles(s.n, seed)], 1)
        return [f[:, c] for f in (e.dfield(), e.ufield(d), e.precond(d)) for c in range(2)]
    u = e.induce()
    if kind == "energy":
        g, vir, parts = e.forces(u)
        eh, gh = e.hal()
        ev, gv = e.valence()
        return dict(grad=g, virial=vir, parts=parts, hal=eh, grad_hal=gh, valence=ev, grad_valence=gv)
    return [u[:, 0], u[:, 1], None] if case.get("learn") else [u[:, 0], u[:, 1]]
