"""Performance cases of the library: the calls a dispersal run makes.

A run builds a meteo term once per meteo interval (kind "meteo"), advances the
concentration step by step ("steps", or operator by operator as the mod_ADS
interface does, "sweeps"; many members at once, "ensemble"), writes its 2-D
products at every output time ("output"), and evaluates settling velocities
point by point ("points") or trains and queries their surrogate
("surrogate").  Stepping passes end with the state read back, as a run does
when it writes its restart file or its 3-D fields.

A case is a dict of plain values.  The state a stepping pass starts from is

  start  an empty domain with the source just switched on
  plume  an eruption under way: puffs of ash drifting and spreading downwind of
         the vent, the coarse bins low and near it, nothing far away from it
  haze   ash everywhere (an old cloud over the whole domain, log-normal, with
         gaps), as the parity tests use

and it goes on from pass to pass, as a run does.  The meteo is the synthetic
one of the workloads: random-phase waves of +-25 m/s with a divergence-free
w, log-normal diffusion, a standard atmosphere, a Suzuki column.  Everything
is made from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from fall3d_b200 import ads, grid as G, source
from fall3d_b200.ads import Domain
from fall3d_b200.ensemble import Ensemble
from fall3d_b200.mlp import SettlingSurrogate

PREC = {"fp64": ads.PREC_FP64, "fp32": ads.PREC_FP32, "fp32c": ads.PREC_FP32C}
F64 = torch.float64
T_ITE = 3600.0
# wet deposition coefficients of the particles, species codes of the bins
WET_A, WET_B = 8.4e-5, 0.79
# the surrogate's training set, batch and refinement
NSAMPLES, BATCH = 1 << 18, 8192


# ---------------------------------------------------------------------------
# the cases
def _steps(name, prec, nx, ny, nz, nb, n, state="plume", lim=2, tm=2, sync=True, wet=False):
    return {"name": name, "kind": "steps", "prec": prec, "nx": nx, "ny": ny, "nz": nz, "nb": nb,
            "n": n, "state": state, "lim": lim, "tm": tm, "sync": sync, "wet": wet}


def listed():
    return [
        # the smallest call: one Euler/minmod step of a tiny domain, latency only
        _steps("step_tiny_fp64", "fp64", 24, 20, 12, 4, 1, "haze", lim=1, tm=1),
        # the classic tephra run in the exact form, from its first step on
        _steps("run_tephra_fp64", "fp64", 100, 80, 40, 6, 100, "start"),
        # a regional run in the exact form
        _steps("run_regional_fp64", "fp64", 200, 150, 40, 8, 40, "plume"),
        # the mod_ADS operators one by one on a ragged grid, exact form, ospre
        {"name": "sweeps_ragged_fp64", "kind": "sweeps", "prec": "fp64", "nx": 157, "ny": 93, "nz": 37,
         "nb": 5, "n": 4, "state": "haze", "lim": 3, "tm": 2},
        # the large domain in the compensated form, an output interval's worth of steps
        _steps("run_large_fp32c", "fp32c", 400, 300, 60, 8, 150, "plume", sync=False),
        # the precision forms on a cloud that fills an odd-sized domain
        _steps("run_haze_fp32", "fp32", 201, 147, 43, 9, 300, "haze", lim=1, sync=False),
        _steps("run_haze_fp32c", "fp32c", 203, 149, 41, 9, 300, "haze", sync=False),
        # every process of a step: wet deposition and radioactive decay after the sweeps
        _steps("run_wet_fp32c", "fp32c", 180, 160, 50, 8, 150, "plume", wet=True),
        # members on uneven grids stepped together on the device clock
        {"name": "ensemble_fp32c", "kind": "ensemble", "prec": "fp32c", "shapes": "60x45x40,100x75x30,150x110x40",
         "members": 9, "nb": 12, "n": 150, "state": "plume", "lim": 2, "tm": 2},
        # once per meteo interval: staggering, K models, settling velocity, CFL time step
        {"name": "meteo_update", "kind": "meteo", "prec": "fp64", "nx": 200, "ny": 150, "nz": 40, "nb": 8,
         "model": 2},
        # an output time: the 2-D products of three species and the mass budget
        {"name": "output_time", "kind": "output", "prec": "fp32c", "nx": 400, "ny": 300, "nz": 60, "nb": 8,
         "state": "plume"},
        # the learned settling velocity: training steps, a gradient, a batch of queries
        {"name": "surrogate", "kind": "surrogate", "n": 500, "npts": 1 << 19, "model": 2},
    ]


def draw(rng):
    """One more case: sizes over the listed ranges, mostly odd ones."""
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["steps"] * 6 + ["sweeps", "ensemble", "ensemble", "meteo", "output", "points", "surrogate"])
    if kind == "points":
        return {"kind": kind, "npts": log(1 << 12, 1 << 20), "model": rng.randint(1, 7)}
    if kind == "surrogate":
        return {"kind": kind, "n": log(50, 600), "npts": log(1 << 14, 1 << 19), "model": rng.randint(1, 7)}
    prec = rng.choice(["fp64", "fp32", "fp32c", "fp32c"])
    nx, ny, nz, nb = log(16, 400), log(12, 300), log(8, 80), rng.randint(1, 16)
    # no more cells than the listed cases of the kind; the exact form costs more
    most = {"steps": 50e6, "sweeps": 4e6, "ensemble": 4e6, "meteo": 9e6, "output": 50e6}[kind]
    if prec == "fp64":
        most = min(most, 9e6)
    while nx * ny * nz * nb > most:
        nx, ny, nz, nb = max(16, int(0.9 * nx)), max(12, int(0.9 * ny)), max(8, int(0.95 * nz)), max(1, nb - 1)
    cost = nx * ny * nz * nb * (2.6e-10 if prec == "fp64" else 2.5e-11)  # of a step, in seconds
    n = max(1, min(log(10, 300), int(0.15 / cost)))
    state = rng.choice(["plume", "plume", "haze", "start"])
    base = {"kind": kind, "prec": prec, "nx": nx, "ny": ny, "nz": nz, "nb": nb}
    if kind == "meteo":
        return dict(base, model=rng.randint(1, 7))
    if kind == "output":
        return dict(base, state=rng.choice(["plume", "haze"]))
    how = {"n": n, "state": state, "lim": rng.randint(1, 3), "tm": rng.choice([1, 2, 2])}
    if kind == "sweeps":
        return dict(base, **dict(how, n=min(n, 8)))
    if kind == "ensemble":
        shapes = ",".join("%dx%dx%d" % (max(8, int(nx * f)), max(8, int(ny * f)), max(6, nz)) for f in (0.6, 1.0))
        return dict({"kind": kind, "prec": prec, "shapes": shapes, "members": rng.randint(2, 8), "nb": nb},
                    **dict(how, n=max(1, n // 4)))
    return dict(base, sync=rng.random() < 0.5, wet=rng.random() < 0.25, **how)


# ---------------------------------------------------------------------------
# inputs
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


class _Rand:
    """Seeded numbers on the device."""

    def __init__(self, seed):
        self.g = torch.Generator(device=_dev())
        self.g.manual_seed(int(seed))

    def uniform(self, lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(shape, generator=self.g, device=_dev(), dtype=F64)

    def normal(self, *shape):
        return torch.randn(shape, generator=self.g, device=_dev(), dtype=F64)

    def one(self, lo=0.0, hi=1.0):
        return float(self.uniform(lo, hi, 1)[0])


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(np.asarray(a, dtype=np.float64)), device=_dev())


def _f(t):
    """A device tensor as a host array in the reference's order (first index fastest)."""
    return t.contiguous().cpu().numpy().T


def _bins(nb):
    phi = np.linspace(-2.0, 6.0, nb) if nb > 1 else np.array([1.0])
    diam = 2.0 ** (-phi) * 1e-3
    rho = 2500.0 - 1500.0 * (phi + 2.0) / 8.0
    cat = np.ones(nb, np.int32)
    spe = np.ones(nb, np.int32)
    if nb >= 6:  # the finest bins are an aerosol and three radionuclides (one Sr90 -> Y90 pair)
        cat[-4:] = (2, 3, 3, 3)
        spe[-4:] = (2, 8, 9, 6)
    return diam, rho, np.full(nb, 0.9), cat, spe


def _grid(nx, ny, nz, h_c=None):
    dl = 0.05
    return G.build_arakawa_c(nx, ny, nz, 10.0, 10.0 + nx * dl, 0.0, ny * dl, 250.0 * nz, G.uniform_sigma(nz), h_c)


def _waves(rnd, g):
    """Corner field (nz+1, ny+1, nx+1) in [-25, 25]: six plane waves of wavenumbers 1..3."""
    dev = _dev()
    X = (torch.arange(g.nx + 1, device=dev, dtype=F64) / g.nx)[None, None, :]
    Y = (torch.arange(g.ny + 1, device=dev, dtype=F64) / g.ny)[None, :, None]
    Z = (torch.arange(g.nz + 1, device=dev, dtype=F64) / g.nz)[:, None, None]
    f = torch.zeros(g.nz + 1, g.ny + 1, g.nx + 1, device=dev, dtype=F64)
    for _ in range(6):
        kx, ky, kz = (int(rnd.one(1, 4)), int(rnd.one(1, 4)), int(rnd.one(0, 2)))
        f += rnd.one(0.5, 1.0) * torch.sin(2 * math.pi * (kx * X + ky * Y + 0.5 * kz * Z) + rnd.one(0, 2 * math.pi))
    f = -25.0 + 50.0 * (f - f.min()) / (f.max() - f.min())
    f[0] = 0.0  # the ground
    return f


def _halo(t):
    return torch.cat([t[..., :1], t, t[..., -1:]], -1)


def _air(z):
    T = 288.15 - 0.0065 * torch.clamp(z, max=11000.0)
    p = 101325.0 * (T / 288.15) ** (9.80665 / (287.05 * 0.0065))
    p = p * torch.exp(-9.80665 * torch.clamp(z - 11000.0, min=0.0) / (287.05 * T))
    return p / (287.05 * T), T


def _meteo_term(rnd, g):
    """Staggered, scaled winds of two snapshots and diffusion, in the step's layouts (first index last)."""
    hm1 = _t(g.Hm1_p)
    us, vs, ws = [], [], []
    for _ in range(2):
        uc, vc = _waves(rnd, g), _waves(rnd, g)
        u = 0.25 * (uc[:-1, :-1] + uc[:-1, 1:] + uc[1:, :-1] + uc[1:, 1:]) / hm1[None, :, None]
        v = 0.25 * (vc[:-1, :, :-1] + vc[:-1, :, 1:] + vc[1:, :, :-1] + vc[1:, :, 1:])
        div = (u[..., 1:] - u[..., :-1]) / _t(g.dX1_b)[1:g.nx + 1] + \
            (v[:, 1:] - v[:, :-1]) / _t(g.dX2_b)[1:g.ny + 1][None, :, None]
        w = torch.zeros(g.nz + 1, g.ny, g.nx, device=u.device, dtype=F64)
        w[1:] = -torch.cumsum(div * _t(g.dX3_b)[1:g.nz + 1][:, None, None], 0)
        us.append(_halo(u))
        vs.append(_halo(v.transpose(1, 2)))
        ws.append(_halo(w.permute(1, 2, 0)))
    k1 = 1500.0 * torch.exp(0.5 * rnd.normal(g.nz, g.ny, g.nx + 4)) / (hm1 * hm1)[None, :, None]
    k2 = 1500.0 * torch.exp(0.5 * rnd.normal(g.nz, g.nx, g.ny + 4))
    k3 = 50.0 * torch.exp(0.5 * rnd.normal(g.ny, g.nx, g.nz + 4))
    return {"u": torch.stack(us), "v": torch.stack(vs), "w": torch.stack(ws), "k1": k1, "k2": k2, "k3": k3}


def _column(g, nb, rate, height, fx=0.35, fy=0.4):
    zs, M = source.suzuki(100, rate, min(height, 0.95 * g.X3max), 4.0, 5.0, 0.0, np.full(nb, 1.0 / nb))
    at = np.full(100, 1.0)
    return source.place_source(g, at * g.lon_p[int(fx * g.nx)], at * g.lat_p[int(fy * g.ny)], zs, M)


def _state(rnd, g, nb, state):
    """Concentration (nb, nz+4, ny+4, nx+4) with zero halos."""
    dev = _dev()
    c = torch.zeros(nb, g.nz + 4, g.ny + 4, g.nx + 4, device=dev, dtype=F64)
    if state == "start":
        return c
    inner = c[:, 2:-2, 2:-2, 2:-2]
    if state == "haze":
        for b in range(nb):
            v = torch.exp(3.0 * rnd.normal(g.nz, g.ny, g.nx) - 2.0)
            m = rnd.uniform(0, 1, g.nz, g.ny, g.nx)
            inner[b] = torch.where(m < 0.15, 0.0, torch.where(m < 0.2, 1e-14, 1e-3 * v / v.max()))
        return c
    npuff, ang = 24, rnd.one(0, 2 * math.pi)
    age = torch.arange(npuff, device=dev, dtype=F64)  # in minutes, about
    x0, y0 = 0.35 * g.nx + 1.0 * age * math.cos(ang), 0.4 * g.ny + 1.0 * age * math.sin(ang)
    x0, y0 = x0 + rnd.uniform(-0.5, 0.5, npuff), y0 + rnd.uniform(-0.5, 0.5, npuff)
    sh = 0.8 + 0.12 * age
    fall = 0.25 * torch.linspace(8.0, 0.05, nb, device=dev, dtype=F64)  # cells a minute
    z0 = 0.6 * min(g.nz, 40) + rnd.uniform(-1, 1, npuff)
    zb = z0[None] - fall[:, None] * age[None]
    amp = rnd.uniform(0.3, 1.0, npuff)[None] * 1e-3 / (sh * sh)[None] * torch.exp(-torch.clamp(-zb, min=0.0))
    gx = torch.exp(-0.5 * ((torch.arange(g.nx, device=dev)[None] - x0[:, None]) / sh[:, None]) ** 2)
    gy = torch.exp(-0.5 * ((torch.arange(g.ny, device=dev)[None] - y0[:, None]) / sh[:, None]) ** 2)
    sz = 2.0 + 0.05 * age
    for b in range(nb):
        gz = torch.exp(-0.5 * ((torch.arange(g.nz, device=dev)[None] - zb[b][:, None]) / sz[:, None]) ** 2)
        inner[b] = torch.einsum("p,pk,pj,pi->kji", amp[b], gz, gy, gx)
    return c


def _vset_levels(g, nb, model=2):
    """(nb, nz+1) settling velocity of the standard atmosphere over flat ground, by the drag-law iteration."""
    diam, rho, psi, cat, _ = _bins(nb)
    rhoa, ta = _air(torch.arange(g.nz + 1, device=_dev(), dtype=F64) * 250.0)
    out = _vset(model, _t(diam)[:, None], _t(rho)[:, None], _t(psi)[:, None], rhoa[None], _visc(ta)[None])
    return torch.where(_t(cat)[:, None] == 2, 0.0, out)


def _cfl(g, m, vs, wind=1.0):
    """Time step of criterion 2 (CFL 0.9) at mid-interval; vs broadcasts to (nb, nz, ny, nx)."""
    nx, ny, nz = g.nx, g.ny, g.nz
    u = wind * 0.5 * (m["u"][0] + m["u"][1])[..., 1:nx + 1]
    v = wind * 0.5 * (m["v"][0] + m["v"][1])[..., 1:ny + 1].transpose(1, 2)
    w = 0.5 * (m["w"][0] + m["w"][1])[..., 1:nz + 1].permute(2, 0, 1)
    k1, k2, k3 = m["k1"][..., 2:nx + 2], m["k2"][..., 2:ny + 2].transpose(1, 2), m["k3"][..., 2:nz + 2].permute(2, 0, 1)
    dx, dy, dz = _t(g.dX1_p)[2:nx + 2], _t(g.dX2_p)[2:ny + 2][:, None], _t(g.dX3_p)[2:nz + 2][:, None, None]
    wm = torch.zeros_like(w)
    for b in range(vs.shape[0]):
        wm = torch.maximum(wm, (w - vs[b]).abs())
    r = 2 * k1 / (dx * dx) + u.abs() / dx + 2 * k2 / (dy * dy) + v.abs() / dy + 2 * k3 / (dz * dz) + wm / dz
    return 0.9 / float(r.max())


class _Inputs:
    """What a stepping program has in hand, from the seed alone."""

    def __init__(self, case, seed, nx, ny, nz):
        rnd = _Rand(seed)
        self.g, self.nb = _grid(nx, ny, nz), case["nb"]
        g = self.g
        self.diam, self.rho, self.psi, self.cat, self.spe = _bins(self.nb)
        self.met = _meteo_term(rnd, g)
        self.vs = _vset_levels(g, self.nb)
        # a pass stays within the meteo interval
        self.dt = min(_cfl(g, self.met, self.vs[:, :nz, None, None]), T_ITE / case.get("n", 1))
        self.ijk, self.vals = _column(g, self.nb, 1e6, 8000.0)
        if case.get("wet"):
            self.pre = torch.clamp(rnd.uniform(-5.0, 20.0, ny, nx), min=0.0)
            self.pblh = rnd.uniform(500.0, 2500.0, ny, nx)
        self.c0 = _state(rnd, g, self.nb, case["state"])
        self.rnd = rnd

    def load(self, dom):
        m = self.met
        dom.set_meteo(*[_f(m[q]) for q in ("u", "v", "w", "k1", "k2", "k3")], None, 0.0, T_ITE)
        rhoc, tc = _air(_t(self.g.z_c.T))
        dom.phys_get_vset(2, _f(rhoc), _f(tc), self.diam, self.rho, self.psi, self.cat)
        dom.set_source(self.ijk, self.vals)
        if hasattr(self, "pre"):
            dom.phys_wet_deposition(WET_A, WET_B, _f(self.pre), _f(self.pblh), self.cat, self.diam)
            if (self.cat == 3).any():
                dom.phys_radionuclides(self.cat, self.spe)


def _buffers(g, nb):
    """The program's own state arrays, page-touched."""
    c = np.zeros((g.nx + 4, g.ny + 4, g.nz + 4, nb), order="F")
    a = np.zeros((g.nx + 4, g.ny + 4, nb), order="F")
    c.fill(0.0)
    a.fill(0.0)
    return c, a


def _members(case, seed):
    """Classes and members of an ensemble case: (inputs per class, [(class, wind factor, source)])."""
    shapes = [tuple(int(v) for v in s.split("x")) for s in case["shapes"].split(",")]
    cls = [_Inputs(case, 10 * seed + q, *s) for q, s in enumerate(shapes)]
    rnd, mem = _Rand(10 * seed + 9), []
    for m in range(case["members"]):
        q = m % len(cls)
        f = 1.0 if m < len(cls) else rnd.one(0.8, 1.2)
        h, rate = rnd.one(6000.0, 10000.0), 1e6 * 2.0 ** rnd.one(-1.0, 1.0)
        mem.append((q, f, _column(cls[q].g, case["nb"], rate, h)))
    return cls, mem


def _corner_meteo(case, seed):
    """Corner fields of a meteo update over hills: two snapshots of winds and virtual temperature."""
    rnd = _Rand(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    X = torch.arange(nx + 1, device=_dev(), dtype=F64)[None, :] / nx
    Y = torch.arange(ny + 1, device=_dev(), dtype=F64)[:, None] / ny
    h = 400.0 * (1.0 + torch.sin(2 * math.pi * (2 * X + Y) + rnd.one(0, 6.0)) * torch.cos(2 * math.pi * (X - 2 * Y)))
    g = _grid(nx, ny, nz, _f(h))
    shape = (nz + 1, ny + 1, nx + 1)
    f = {"uc": [_waves(rnd, g) for _ in range(2)], "vc": [_waves(rnd, g) for _ in range(2)],
         "wc": [rnd.uniform(-0.4, 0.4, *shape) for _ in range(2)]}
    z = _t(g.z_c.T)
    f["rhoc"], f["tc"] = _air(z)
    f["tvc"] = [f["tc"] + 0.006 * z + rnd.uniform(-1.0, 1.0, *shape) for _ in range(2)]
    f["pblh"] = rnd.uniform(300.0, 2500.0, ny, nx)
    f["mon"] = rnd.uniform(20.0, 400.0, ny, nx) * torch.where(rnd.uniform(0, 1, ny, nx) < 0.5, -1.0, 1.0)
    f["ust"] = rnd.uniform(0.05, 0.8, ny, nx)
    return g, f


def _points(rnd, n):
    """Particles and air: diameter 1 um - 4 mm (log-uniform), density, sphericity, air density, viscosity."""
    d = torch.exp(rnd.uniform(math.log(1e-6), math.log(4e-3), n))
    return [d, rnd.uniform(800.0, 3000.0, n), rnd.uniform(0.5, 1.0, n), rnd.uniform(0.1, 1.3, n),
            rnd.uniform(1.35e-5, 1.8e-5, n)]


def _species(nb):
    """Bins of the output fields: all tephra, the fine tephra, one more species."""
    spe = _bins(nb)[4]
    tephra = [b for b in range(nb) if spe[b] == 1]
    return [tephra, tephra[len(tephra) // 2:], [nb - 1]]


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case, kind = case, case["kind"]
    if kind in ("steps", "sweeps", "output"):
        inp = _Inputs(case, seed, case["nx"], case["ny"], case["nz"])
        s.dt, s.nb = inp.dt, inp.nb
        s.dom = Domain(inp.g, inp.nb, case.get("lim", 2), case.get("tm", 2), PREC[case["prec"]])
        inp.load(s.dom)
        s.dom.upload_state(_f(inp.c0), None)
        s.c, s.a = _buffers(inp.g, inp.nb)
        if kind == "output":  # the ground deposit of the run so far, and the corner heights
            s.a[2:-2, 2:-2, :] = _f(inp.rnd.uniform(0.0, 1.0, inp.nb, case["ny"], case["nx"]))
            s.dom.upload_state(None, s.a)
            s.dom.nc_IO_out_res([0])
    elif kind == "ensemble":
        cls, mem = _members(case, seed)
        s.ens = Ensemble([c.g for c in cls], case["nb"], [m[0] for m in mem], [m[1] for m in mem], case["lim"],
                         case["tm"], PREC[case["prec"]])
        for q, c in enumerate(cls):
            s.ens.set_class_meteo(q, *[_f(c.met[k]) for k in ("u", "v", "w", "k1", "k2", "k3")], None, 0.0, T_ITE)
            rhoc, tc = _air(_t(c.g.z_c.T))
            s.ens.compute_class_vset(q, 2, _f(rhoc), _f(tc), c.diam, c.rho, c.psi, c.cat)
        host = [_f(c.c0) for c in cls]
        for m, (q, _, src) in enumerate(mem):
            s.ens.set_member_source(m, *src)
            s.ens.upload_member_state(m, host[q], None)
        s.ens.compute_time_steps(0.5, run_end=T_ITE / case["n"])
    elif kind == "meteo":
        g, f = _corner_meteo(case, seed)
        s.dom = Domain(g, case["nb"], precision=PREC[case["prec"]])
        s.dom.set_terrain()
        s.f = {k: [_f(x) for x in v] if isinstance(v, list) else _f(v) for k, v in f.items()}
        s.bins = _bins(case["nb"])
    elif kind == "points":
        s.pts = [x.cpu().numpy() for x in _points(_Rand(seed), case["npts"])]
    elif kind == "surrogate":
        rnd = _Rand(seed)
        s.mlp = SettlingSurrogate(model=case["model"], seed=seed)
        s.mlp.generate(NSAMPLES, seed=seed + 1)
        s.p0 = s.mlp.params
        s.seed = seed
        s.pts = [x.cpu().numpy() for x in _points(rnd, case["npts"])]
        s.feat, s.targ, s.weights = _gradient_inputs(seed)
    return s


def _gradient_inputs(seed):
    rnd = _Rand(seed + 5)
    feat = rnd.uniform(-1.0, 1.0, 1 << 15, 5).float().cpu().numpy()
    targ = rnd.uniform(-1.0, 0.0, 1 << 15).float().cpu().numpy()
    return feat, targ, (0.2 * rnd.normal(4609)).float().cpu().numpy()


# ---------------------------------------------------------------------------
# one pass
def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "steps":
        f, t = np.zeros(6), 0.0
        for it in range(case["n"]):
            if case["sync"]:
                s.dom.F3D_time_step(s.dt, t, it, f)
            else:
                s.dom.step_async(s.dt, t, it)
            t += s.dt
        if not case["sync"]:
            s.dom.get_fluxes(f)
        out = {"fluxes": f}
        out["c"], out["acum"] = s.dom.download_state(s.c, s.a)
        if case["wet"]:
            out["awet"] = s.dom.get_awet()
        return out
    if kind == "sweeps":
        fx, t = [0.0] * 6, 0.0
        for it in range(case["n"]):
            st = t / T_ITE
            s.dom.ADS_update_horizontal_vcomps(st)
            s.dom.add_source(s.dt)
            fx[0], fx[1] = s.dom.ADS_solve_along_x(s.dt, fx[0], fx[1])
            fx[2], fx[3] = s.dom.ADS_solve_along_y(s.dt, fx[2], fx[3])
            fx[5], fx[4] = s.dom.ADS_solve_along_z(s.dt, st, fx[5], fx[4])
            t += s.dt
        c, a = s.dom.download_state(s.c, s.a)
        return {"c": c, "acum": a, "fluxes": np.array(fx)}
    if kind == "ensemble":
        s.ens.set_clock(0.0, 0)
        s.ens.run(case["n"])
        out = {"fluxes": s.ens.get_fluxes()}
        for m in range(s.ens.nm):
            out["c%d" % m], out["acum%d" % m] = s.ens.download_member_state(m)
        return out
    if kind == "meteo":
        f = s.f
        s.dom.set_meteo_corners_kdiffu(f["uc"], f["vc"], f["wc"], 2, 3, 0.5, tvc_pair=f["tvc"], pblh=f["pblh"],
                                       mon=f["mon"], ust=f["ust"], t_its=0.0, t_ite=T_ITE)
        diam, rho, psi, cat, _ = s.bins
        vs = s.dom.phys_get_vset(case["model"], f["rhoc"], f["tc"], diam, rho, psi, cat, want_host=True)
        return {"vs": vs, "dt": s.dom.grid_get_time_step(0.5)[1]}
    if kind == "output":
        out = {"mass": s.dom.grid_get_mass_volume(per_bin=True)[1]}
        for q, bins in enumerate(_species(s.nb)):
            out["species%d" % q] = s.dom.nc_IO_out_res(bins)
        return out
    if kind == "points":
        v, flags = ads.phys_get_vset_point(*s.pts, model=case["model"])
        return {"v": v, "flags": flags}
    s.mlp.params = s.p0
    loss, _ = s.mlp.train(steps=case["n"], batch=BATCH, seed=s.seed + 2)
    trained = s.mlp.params
    v, used = s.mlp.predict(*s.pts, refine=1)
    s.mlp.params = s.weights
    grad, gloss = s.mlp.gradient(s.feat, s.targ)
    return {"grad": grad, "grad_loss": float(gloss), "loss": loss, "params": trained, "v": v, "used": used}


# ---------------------------------------------------------------------------
# what a pass cannot do without
def work(case):
    """Inputs read once and outputs written once, and the scheme's arithmetic over the whole domain: a sweep
    is about 27 operations a cell and Runge-Kutta stage, three sweeps a step."""
    kind = case["kind"]
    if kind == "points":
        return {"bytes": 52.0 * case["npts"], "flops": 400.0 * case["npts"]}
    if kind == "surrogate":
        layer = 2.0 * 4544
        return {"bytes": 32.0 * BATCH * case["n"] + 52.0 * case["npts"],
                "flops": 3 * layer * (BATCH * case["n"] + (1 << 15)) + layer * case["npts"]}
    word = {"fp64": 8, "fp32": 4, "fp32c": 8}[case["prec"]]
    nb = case["nb"]
    if kind == "ensemble":
        shapes = [tuple(int(v) for v in q.split("x")) for q in case["shapes"].split(",")]
        cells = float(sum(np.prod(shapes[m % len(shapes)]) for m in range(case["members"])))
        faces = float(sum(np.prod(q) for q in shapes))
    else:
        cells = faces = float(case["nx"] * case["ny"] * case["nz"])
    if kind == "meteo":
        return {"bytes": 8.0 * cells * (10 + nb), "flops": cells * (150 + 400 * nb)}
    if kind == "output":
        bins = sum(len(b) for b in _species(nb))
        return {"bytes": cells * word * nb, "flops": 14.0 * cells * bins}
    stages = 4 if case["tm"] == 2 else 1
    # the state and the meteo term in, the state out and on the host in 64 bits
    return {"bytes": cells * nb * (2.0 * word + 8.0) + faces * (9.0 + nb) * (8 if case["prec"] == "fp64" else 4),
            "flops": case["n"] * cells * nb * 3.0 * 27.0 * stages}


# ---------------------------------------------------------------------------
# 64-bit values
def _visc(t):
    return 1.827e-5 * ((291.15 + 120.0) / (t + 120.0)) * (t / 291.15) ** 1.5


def _vset(model, d, rhop, psi, rhoa, mu):
    """Fixed-point settling velocity (phys_get_vset_point), elementwise."""
    d, rhop, psi, rhoa, mu = torch.broadcast_tensors(d, rhop, psi, rhoa, mu)
    if model == 4:
        return 1.2065 * mu * (d ** 3 * 9.81 * rhop * rhoa * psi ** 1.6 / (mu * mu)) ** 0.5206 / (d * rhoa)
    k1 = 3.0 / (1.0 + 2.0 / torch.sqrt(psi))
    k2 = 10.0 ** (1.8148 * (-torch.log10(psi)) ** 0.5743)
    wilson = 2.0 * torch.sqrt(1.07 - psi)
    cd100 = 0.24 * psi ** -0.828 + wilson
    pa = (1.0 - cd100) / 900.0

    def cd_of(re):
        if model == 1:
            return torch.where(re <= 988.947, 24.0 / re * (1.0 + 0.15 * re ** 0.687), 0.44)
        if model == 2:
            x = re * k1
            return 24.0 / x * (1.0 + 0.1118 * (x * k2) ** 0.6567) + 0.4305 * k2 / (1.0 + 3305.0 / (x * k2))
        if model == 3:
            return 24.0 / re * psi ** -0.828 + wilson
        if model == 5:
            return torch.where(re <= 100.0, 24.0 / re * psi ** -0.828 + wilson,
                               torch.where(re < 1000.0, pa * re + (1.0 - 1000.0 * pa), 1.0))
        if model == 6:
            c = 24.0 * (1.0 + 0.15 * re ** 0.687) / re + 0.42 / (1.0 + 42500.0 / re ** 1.16)
            return 0.74533 * re ** 0.146012 * c / psi ** (0.5134 / torch.clamp(re, min=0.01) ** 0.2)
        return 24.0 / re * (((1.0 - psi) / re + 1.0) ** 0.25 + 0.1806 * re ** 0.6459 * psi ** (-(re ** 0.08))) + \
            0.4251 / (1.0 + 6880.95 / re * psi ** 5.03)

    base = 4.0 * 9.81 * d * rhop / 3.0
    v = torch.sqrt(base / rhoa)
    live = torch.ones_like(v, dtype=torch.bool)
    for _ in range(1000):
        new = torch.sqrt(base / (cd_of(rhoa * v * d / mu) * rhoa))
        done = (new - v).abs() <= 1e-12 + 1e-6 * new.abs()
        v = torch.where(live, new, v)
        live &= ~done
        if not bool(live.any()):
            break
    return v


def _rhs(a, u, kk, dxp, dxb, lim):
    """KT right-hand side along the last axis of a (two ghosts at each end), and the end fluxes F + P."""
    n = a.shape[-1] - 4
    d = a[..., 1:] - a[..., :-1]
    d1, d0 = d[..., :-1], d[..., 1:]
    flat, still = d0.abs() < 1e-12, d1.abs() < 1e-12
    r = d1 / torch.where(flat, 1.0, d0)
    if lim == 1:
        r = torch.where(flat, 1.0, torch.clamp(r, 0.0, 1.0))
    elif lim == 2:
        r = torch.maximum(torch.clamp(2.0 * r, max=1.0), torch.clamp(r, max=2.0)).clamp_(min=0.0)
        r = torch.where(flat, torch.where(still, 0.0, 2.0), r)
    else:
        q = r * r + r
        r = torch.where(flat, torch.where(still, 0.0, 1.5), 1.5 * q / (q + 1.0))
    h = 0.5 * r * d0
    cl = a[..., 1:n + 2] + h[..., :n + 1]
    cr = a[..., 2:n + 3] - h[..., 1:n + 2]
    F = 0.5 * u * (cl + cr) - 0.5 * u.abs() * (cr - cl)
    P = kk * d[..., 1:n + 2] / dxp
    W = P - F
    ends = (F[..., 0] + P[..., 0], F[..., -1] + P[..., -1])
    return (W[..., 1:] - W[..., :-1]) / dxb, ends


def _sweep(c, u, kk, dxp, dxb, dt, lim, tm):
    """One operator along the last axis: the new values and the fluxes at both ends."""
    gl = torch.where(u[..., :1] > 0.0, -c[..., :1], c[..., :1])
    gr = torch.where(u[..., -1:] < 0.0, -c[..., -1:], c[..., -1:])

    def pad(x):
        return torch.cat([gl, gl, x, gr, gr], -1)

    k1, ends = _rhs(pad(c), u, kk, dxp, dxb, lim)
    if tm == 1:
        return c + dt * k1, ends
    new = c + dt / 6.0 * k1
    k, _ = _rhs(pad(c + 0.5 * dt * k1), u, kk, dxp, dxb, lim)
    new += dt / 3.0 * k
    k, _ = _rhs(pad(c + 0.5 * dt * k), u, kk, dxp, dxb, lim)
    new += dt / 3.0 * k
    k, ends = _rhs(pad(c + dt * k), u, kk, dxp, dxb, lim)
    return new + dt / 6.0 * k, ends


class _Model:
    """The scheme in 64-bit torch for one domain."""

    def __init__(self, inp, dt, wind=1.0, src=None):
        g, m = inp.g, inp.met
        self.g, self.nb, self.dt, self.wind, self.m, self.vs = g, inp.nb, dt, wind, m, inp.vs
        self.c = inp.c0[:, 2:-2, 2:-2, 2:-2].clone()
        self.acum = torch.zeros(self.nb, g.ny, g.nx, device=self.c.device, dtype=F64)
        self.awet = torch.zeros_like(self.acum)
        self.flux = np.zeros(6)
        ijk, vals = src if src is not None else (inp.ijk, inp.vals)
        ijk = np.asarray(ijk, np.int64).reshape(-1, 3) - 1
        vol = g.dX1_p[ijk[:, 0] + 2] * g.dX2_p[ijk[:, 1] + 2] * g.dX3_p[ijk[:, 2] + 2] * (
            g.Hm1_p[ijk[:, 1]] * g.Hm2_p[ijk[:, 1] + 2] * g.Hm3_p[ijk[:, 0], ijk[:, 1]])
        self.src = [torch.as_tensor(q, device=self.c.device) for q in (ijk[:, 2], ijk[:, 1], ijk[:, 0])]
        self.add = _t((vals / vol[:, None]).T)
        b1, b2, b3 = (_t(x)[1:-2] for x in (g.dX1_b, g.dX2_b, g.dX3_b))  # of cell p
        p1, p2, p3 = (_t(x)[1:-2] for x in (g.dX1_p, g.dX2_p, g.dX3_p))  # below face f
        self.axis = {
            "x": (lambda c: c, m["u"], m["k1"], p1, b1, b3[:, None] * b2[None], (0, 1)),
            "y": (lambda c: c.transpose(-1, -2), m["v"], m["k2"], p2, b2, b3[:, None] * b1[None], (2, 3)),
            "z": (lambda c: c.permute(0, 2, 3, 1), m["w"], m["k3"], p3, b3, b2[:, None] * b1[None], (5, 4)),
        }

    def source(self):
        k, j, i = self.src
        self.c[:, k, j, i] += self.dt * self.add

    def sweep(self, ax, st, lim, tm):
        view, vel, kk, dxp, dxb, area, (lo, hi) = self.axis[ax]
        u = (1.0 - st) * vel[0] + st * vel[1]
        u = u[..., 1:-1] * (1.0 if ax == "z" else self.wind)
        k = 0.5 * (kk[..., 1:-2] + kk[..., 2:-1])
        group = max(1, int(4e6 // self.c[0].numel()))
        for b in range(0, self.nb, group):
            part = view(self.c[b:b + group])
            vel_b = u[None] if ax != "z" else u[None] - self.vs[b:b + group][:, None, None, :]
            new, (f0, f1) = _sweep(part.contiguous(), vel_b, k[None], dxp, dxb, self.dt, lim, tm)
            part.copy_(new)
            self.flux[lo] += float((f0 * area).sum()) * self.dt
            self.flux[hi] += float((f1 * area).sum()) * self.dt
            if ax == "z":
                self.acum[b:b + group] += f0.abs() * self.dt

    def step(self, it, time, lim, tm):
        st = time / T_ITE
        self.source()
        for ax in ("xyz" if it % 2 == 0 else "yxz"):
            self.sweep(ax, st, lim, tm)

    def after(self, inp):
        """Wet deposition below the boundary-layer top, then decay with the Sr90 -> Y90 assignment."""
        g = self.g
        lam = torch.clamp(self.dt * WET_A * inp.pre ** WET_B, max=1.0)
        zc = _t(g.z_c.T)
        zl = 0.25 * (zc[:, :-1, :-1] + zc[:, 1:, :-1] + zc[:, :-1, 1:] + zc[:, 1:, 1:])
        below = 0.5 * (zl[1:] + zl[:-1]) <= inp.pblh[None]
        dz = _t(g.dX3_p)[2:g.nz + 2][:, None, None]
        for b in range(self.nb):
            if inp.cat[b] in (1, 3) and inp.diam[b] <= 1e-4:
                out = torch.where(below, lam[None] * self.c[b], 0.0)
                self.awet[b] += (dz * out).sum(0)
                self.c[b] -= out
        rate = {6: 9.29e-10, 8: 7.63e-10, 9: 2.98e-6}
        for b in range(self.nb):
            if inp.cat[b] != 3:
                continue
            for x in (self.c, self.acum, self.awet):
                x[b] *= math.exp(-rate[int(inp.spe[b])] * self.dt)
                if inp.spe[b] == 9:  # set from the parent, the bin before
                    x[b] = x[b - 1] * (1.0 - math.exp(-rate[8] * self.dt))

    def arrays(self, ghosts=True):
        """The state in the layout of a download: halo-inclusive; a domain's has zero-gradient face ghosts, a
        member's zeros there."""
        c, a = _buffers(self.g, self.nb)
        x = _f(self.c)
        c[2:-2, 2:-2, 2:-2] = x
        for h, e in ((0, 0), (1, 0), (-2, -1), (-1, -1)) if ghosts else ():
            c[h, 2:-2, 2:-2] = x[e]
            c[2:-2, h, 2:-2] = x[:, e]
            c[2:-2, 2:-2, h] = x[:, :, e]
        a[2:-2, 2:-2] = _f(self.acum)
        return c, a


def _corner_model(case, seed):
    """The meteo update in 64-bit torch: settling velocity and time step."""
    g, f = _corner_meteo(case, seed)
    nx, ny, nz, nb = g.nx, g.ny, g.nz, case["nb"]
    diam, rho, psi, cat, _ = _bins(nb)

    def mean4(a):  # over the corners of a horizontal cell
        return 0.25 * (a[:, :-1, :-1] + a[:, :-1, 1:] + a[:, 1:, :-1] + a[:, 1:, 1:])

    hm1, hm3 = _t(g.Hm1_p)[:, None], _t(g.Hm3_p.T)
    rhoa, mu = mean4(f["rhoc"]), _visc(mean4(f["tc"]))
    vs = torch.zeros(nb, nz + 3, ny, nx, device=rhoa.device, dtype=F64)
    for b in range(nb):
        if cat[b] != 2:
            vs[b, 1:-1] = _vset(case["model"], *(_t(q[b]) for q in (diam, rho, psi)), rhoa, mu) / hm3
        vs[b, 0], vs[b, -1] = vs[b, 1], vs[b, -2]
    sx, sy = _t(g.dhdx_p.T), _t(g.dhdy_p.T)
    decay = 1.0 - _t(g.X3_c)[:, None, None] / g.X3max
    us, vv, ws = [], [], []
    for s in range(2):
        uc, vc, wc = (f[q][s].clone() for q in ("uc", "vc", "wc"))
        wc[0] = 0.0
        us.append(_halo(0.25 * (uc[:-1, :-1] + uc[:-1, 1:] + uc[1:, :-1] + uc[1:, 1:]) / hm1[None]))
        v = 0.25 * (vc[:-1, :, :-1] + vc[:-1, :, 1:] + vc[1:, :, :-1] + vc[1:, :, 1:])
        vv.append(_halo(v.transpose(1, 2)))
        w = (mean4(wc) - sx * decay * mean4(uc) - sy * decay * mean4(vc)) / hm3
        ws.append(_halo(w.permute(1, 2, 0)))
    # diffusion from the corner fields at mid-interval
    u, v, tv = (0.5 * (f[q][0] + f[q][1]) for q in ("uc", "vc", "tvc"))
    dx, dy = (_t(g.dX1_p)[2:-2][None, :] * hm1), _t(g.dX2_p)[2:-2][:, None]

    def slope(a):
        a = a[:-1]
        x = 0.5 * (a[:, :-1, 1:] - a[:, :-1, :-1] + a[:, 1:, 1:] - a[:, 1:, :-1]) / dx
        y = 0.5 * (a[:, 1:, :-1] - a[:, :-1, :-1] + a[:, 1:, 1:] - a[:, :-1, 1:]) / dy
        return x, y

    (ux, uy), (vx, vy) = slope(u), slope(v)
    kt = 0.28 * 0.28 * dx * dy * torch.sqrt((ux - vy) ** 2 + (vx + uy) ** 2)
    kn = 8000.0 * (0.036 / (hm1 * g.dlon)) * (0.036 / g.dlat)
    kh = torch.where((kt < 1.0) & (kn < 1.0), 100.0, torch.clamp(kt * kn / (kt + kn), min=100.0))
    zc, hp = _t(g.z_c.T), mean4(_t(g.h_c.T)[None])[0]
    zl = mean4(zc) - hp
    z = torch.clamp(0.5 * (zl[1:] + zl[:-1]), min=0.0)
    zol = z / f["mon"]
    fih = torch.where(zol < 0.0, 1.0 / torch.sqrt(torch.clamp(1.0 - 15.0 * zol, min=1.0)), 1.0 + 5.0 * zol)
    low = torch.clamp(0.4 * z * f["ust"] * (1.0 - z / f["pblh"]) ** 2 / fih, min=0.0)
    lc = 1.0 / (1.0 / (0.4 * z) + 1.0 / 30.0)
    mod = torch.sqrt(mean4(u) ** 2 + mean4(v) ** 2)
    t4, dz = mean4(tv), zl[1:] - zl[:-1]
    um2 = torch.clamp((0.5 * (mod[1:] + mod[:-1])) ** 2, min=1e-18)
    ri = 9.81 * dz * (t4[1:] - t4[:-1]) / (um2 * 0.5 * (t4[1:] + t4[:-1]))
    fc = torch.where(ri > 0.0, 1.0 / (1.0 + 10.0 * ri * (1.0 + 8.0 * ri)),
                     torch.sqrt(torch.clamp(1.0 - 18.0 * ri, min=0.0)))
    high = torch.clamp(lc * lc * ((mod[1:] - mod[:-1]) / dz).abs() * fc, min=0.0)
    k3 = torch.where(z < f["pblh"], low, high)
    dec = 1.0 - _t(g.X3_p)[:, None, None] / g.X3max
    k3 = (k3 + (sx * dec) ** 2 * kh + (sy * dec) ** 2 * kh) / (hm3 * hm3)
    m = {"u": torch.stack(us), "v": torch.stack(vv), "w": torch.stack(ws), "k1": _halo(_halo(kh / (hm1 * hm1))),
         "k2": _halo(_halo(kh.transpose(1, 2))), "k3": _halo(_halo(k3.permute(1, 2, 0)))}
    return {"vs": _f(vs), "dt": _cfl(g, m, vs[:, 1:nz + 1])}


def _output_model(case, seed):
    """The 2-D products and the mass per bin in 64-bit torch; the run keeps no boundary halo."""
    inp = _Inputs(case, seed, case["nx"], case["ny"], case["nz"])
    g, nb = inp.g, inp.nb
    acum = inp.rnd.uniform(0.0, 1.0, nb, g.ny, g.nx)
    c = inp.c0
    vol = (_t(g.dX3_p)[2:-2][:, None, None] * _t(g.dX2_p)[2:-2][:, None]) * _t(g.dX1_p)[2:-2]
    out = {"mass": np.array([float((c[b, 2:-2, 2:-2, 2:-2] * vol).sum()) for b in range(nb)])}
    zc = _t(g.z_c.T)
    metric = (_t(g.Hm1_p) * _t(g.Hm2_p)[2:-2])[:, None] * _t(g.Hm3_p.T)
    edge = torch.nn.functional.pad(acum[None], (1, 1, 1, 1), mode="replicate")[0]
    ac = 0.25 * (edge[:, :-1, :-1] + edge[:, 1:, :-1] + edge[:, :-1, 1:] + edge[:, 1:, 1:])
    both = (slice(None, -1), slice(1, None))
    for q, bins in enumerate(_species(nb)):
        w = torch.zeros_like(zc)
        for b in bins:
            x = c[b, 1:-1, 1:-1, 1:-1].clone()
            x[1:-1, 1:-1, 1:-1] *= 1e3 / metric
            x = torch.clamp(x, min=0.0)
            w += sum(x[i, j, k] for i in both for j in both for k in both) / 8.0
        dz = zc[1:] - zc[:-1]
        level = torch.arange(g.nz + 1, device=w.device)[:, None, None]
        top = torch.where(w > 50e-6, level, -1).amax(0)
        height = torch.where(top >= 0, zc.gather(0, top.clamp(min=0)[None])[0], 0.0)
        out["species%d" % q] = {"con_sur": _f(w[0]), "col_mass": _f((0.5 * (w[1:] + w[:-1]) * dz).sum(0)),
                                "cloud_top": _f(height),
                                "grn_load": _f(sum(ac[b] for b in bins) + torch.zeros_like(w[0]))}
    return out


def _gradient_model(seed):
    """Mean squared error of the 5-64-64-1 tanh network and its gradient, by autograd in 64 bits."""
    feat, targ, par = _gradient_inputs(seed)
    p = torch.tensor(par, device=_dev(), dtype=F64, requires_grad=True)
    w1, b1, w2, b2, w3, b3 = torch.split(p, [320, 64, 4096, 64, 64, 1])
    h = torch.tanh(_t(feat) @ w1.view(64, 5).T + b1)
    h = torch.tanh(h @ w2.view(64, 64).T + b2)
    loss = ((h @ w3 + b3 - _t(targ)) ** 2).mean()
    loss.backward()
    return {"grad": p.grad.cpu().numpy(), "grad_loss": float(loss.detach())}


def exact(case, seed):
    """What run() returns on a new state, in 64 bits; the trained weights and what follows from them have no
    such value."""
    kind = case["kind"]
    if kind == "points":
        v = _vset(case["model"], *_points(_Rand(seed), case["npts"]))
        return {"v": v.cpu().numpy(), "flags": None}
    if kind == "surrogate":
        return dict(_gradient_model(seed), loss=None, params=None, v=None, used=None)
    if kind == "meteo":
        return _corner_model(case, seed)
    if kind == "output":
        return _output_model(case, seed)
    if kind == "ensemble":
        cls, mem = _members(case, seed)
        out, fl = {}, []
        for m, (q, wind, src) in enumerate(mem):
            inp = cls[q]
            dt = min(_cfl(inp.g, inp.met, inp.vs[:, :inp.g.nz, None, None], wind), T_ITE / case["n"])
            M = _Model(inp, dt, wind, src)
            for it in range(case["n"]):
                M.step(it, it * M.dt, case["lim"], case["tm"])
            out["c%d" % m], out["acum%d" % m] = M.arrays(ghosts=False)
            fl.append(M.flux)
        return dict(out, fluxes=np.stack(fl))
    inp = _Inputs(case, seed, case["nx"], case["ny"], case["nz"])
    M = _Model(inp, inp.dt)
    for it in range(case["n"]):
        if kind == "sweeps":  # x, y, z at every step
            M.source()
            for ax in "xyz":
                M.sweep(ax, it * M.dt / T_ITE, case["lim"], case["tm"])
        else:
            M.step(it, it * M.dt, case["lim"], case["tm"])
            if case["wet"]:
                M.after(inp)
    out = {"fluxes": M.flux}
    out["c"], out["acum"] = M.arrays()
    if case.get("wet"):
        w = np.zeros_like(out["acum"])
        w[2:-2, 2:-2] = _f(M.awet)
        out["awet"] = w
    return out
