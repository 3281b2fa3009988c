"""Performance cases of the anelastic core: time-stepping runs, an ensemble and
adjoints through the package's public entry points (model_gb300.anelastic).

A pass is what a caller's time loop does between two looks at the state: one
or a few steps (Model.step, Ensemble.step) or one gradient (Model.adjoint).
Model states stay on the GPU and are handed out as tensors over the library's
buffers; ensembles and adjoints have host access only, so their passes include
the download of the results.

`exact` restates the nonlinear step (advection, pressure solve, boundary
conditions, Kessler) in 64 bits with torch, for the kinds that run no more
than that.
"""
import dataclasses
import functools
import math

import numpy as np
import torch

from model_gb300 import abi, anelastic, configs

PROG = abi.PROG_NAMES
ICE = ("qs", "qi")


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _case(name, kind, nx, ny, nz, steps, f32=True, **kw):
    c = {"name": name, "kind": kind, "nx": nx, "ny": ny, "nz": nz, "steps": steps, "f32": f32, "tuned": False}
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call: a coupled model that takes the state after every single step (the dry bubble's grid)
        _case("bubble_one_step", "bubble", 64, 64, 40, 1),
        # the warm-rain thunderstorm, the usual job, autotuned once as a long run does
        _case("storm", "storm", 128, 128, 48, 10, tuned=True),
        # the same in double precision, the parity path
        _case("storm_f64", "storm", 128, 128, 48, 2, f32=False),
        # with the optional physics: 4th-order diffusion, turbulence and ocean fluxes
        _case("storm_physics", "physics", 128, 128, 48, 4),
        # jet and vortex of the monsoon grid: a basic state that varies horizontally.  At 40 km spacing the pressure's
        # long waves need double precision
        _case("jet_f64", "jet", 192, 128, 32, 1, f32=False),
        # the ice scheme, a deep cloud of all five water species
        _case("ice_cloud", "ice", 128, 128, 48, 2),
        # the hydrostatic set on the thunderstorm grid at 2 km
        _case("hydrostatic", "hydro", 128, 128, 48, 4),
        # a ragged periodic channel with semi-Lagrangian rain: odd and prime transform lengths, odd level count
        _case("channel_odd", "channel", 101, 75, 33, 2),
        # an uneven ensemble: members of two sizes advanced together, then downloaded
        _case("ensemble", "ensemble", 96, 96, 40, 20, members=6, nx2=160, ny2=160, nz2=48, members2=2, tuned=True),
        # the squall line, the largest single domain
        _case("squall_line", "squall", 512, 512, 64, 2, tuned=True),
        # a dry gradient in single precision: forward, recompute, adjoint, download
        _case("adjoint_bubble", "adjoint_dry", 64, 64, 40, 20, every=5),
        # a moist gradient in double precision on a small storm
        _case("adjoint_storm_f64", "adjoint_moist", 64, 64, 32, 6, every=3, f32=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["bubble", "storm", "storm", "storm_f64", "physics", "jet", "ice", "hydro", "channel",
                       "ensemble", "squall", "adjoint_dry", "adjoint_moist"])
    f32 = kind not in ("storm_f64", "adjoint_moist", "jet")
    kind = "storm" if kind == "storm_f64" else kind
    lo, hi = {"bubble": (32, 96), "squall": (192, 448), "channel": (40, 160), "ensemble": (40, 128),
              "adjoint_dry": (40, 128), "adjoint_moist": (32, 80)}.get(kind, (40, 256 if f32 else 144))

    def width():
        n = _log_int(rng, lo, hi)
        # most grids have even, smooth sizes; some are whatever the domain gave
        return n if rng.random() < 0.35 else max(lo, 8 * int(round(n / 8)))

    nx, ny = width(), width()
    nz = rng.choice([24, 32, 33, 40, 44, 48, 50, 64] + ([96] if kind != "squall" else []))
    if kind == "hydro":
        nz = rng.choice([24, 32, 33, 40, 44, 48, 50])
    if kind == "channel":
        nz = rng.choice([24, 31, 33, 40])
    if kind.startswith("adjoint"):
        nz = rng.choice([24, 32, 40])
    steps = rng.choice([1, 2, 3, 4, 6])
    kw = {}
    if kind in ("ice", "squall", "jet"):
        steps = rng.choice([1, 2])
    if kind == "ensemble":
        steps = rng.choice([10, 20])
        kw = {"members": rng.randint(2, 6), "nx2": width(), "ny2": width(), "nz2": rng.choice([32, 40, 48]),
              "members2": rng.randint(1, 2)}
    if kind.startswith("adjoint"):
        steps = rng.choice([8, 12, 16] if f32 else [2, 4])
        kw = {"every": rng.choice([2, 4])}
    c = _case("", kind, nx, ny, nz, steps, f32=f32, **kw)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs: a workload's settings and basic state, with a seeded perturbation
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=4)
def _basic(kind, nx, ny, nz):
    """Settings and noise-free state of a kind (shared by its seeds)."""
    dz = max(200.0, round(19200.0 / nz, -1))
    if kind in ("bubble", "adjoint_dry"):
        return configs.dry_bubble(nx=nx, ny=ny, nz=nz, noise=0.0)
    if kind == "jet":
        return configs.jet_vortex(nx=nx, ny=ny, nz=nz)
    if kind == "squall":
        return configs.squall_line(nx=nx, ny=ny, nz=nz)
    if kind == "ice":
        return configs.ice_cloud(nx=nx, ny=ny, nz=nz, dz=max(dz, 400.0))
    if kind == "channel":
        return configs.moist_blob(nx=nx, ny=ny, nz=nz, rain_fallout=2, periodic=1)
    wl = configs.thunderstorm(nx=nx, ny=ny, nz=nz, dz=dz, dx=2000.0 if kind == "hydro" else 1000.0, noise=0.0)
    if kind == "hydro":
        wl.hydrostatic, wl.dt = 1, 2.0
    elif nz > 64:
        wl.dt = 2.0
    if kind == "physics":
        wl.use_explicit_diffusion, wl.turbulence_option, wl.use_surface_heat_flux = 1, 1, 1
    return wl


def _state(kind, nx, ny, nz, seed):
    """The workload with seeded perturbations: noise on theta and the winds,
    the anomaly's strength, and (moist kinds) a cloud with rain in it."""
    base = _basic(kind, nx, ny, nz)
    rng = np.random.default_rng(seed)
    f = dict(base.fields)
    n3 = (nx, ny, nz)

    def noise(amp):
        r = rng.random(n3, dtype=np.float32).astype(np.float64)
        r -= 0.5
        r *= 2.0 * amp
        r[:, :, 0] = 0.0
        r[:, :, -1] = 0.0
        return r

    f["th"] = f["th"] * (0.8 + 0.4 * rng.random()) + noise(0.05)
    f["u"] = f["u"] + noise(0.1)
    f["v"] = f["v"] + noise(0.1)
    f["w"] = f["w"] + noise(0.02)
    if base.microphysics_option:
        if kind not in ("ice", "channel"):
            x = (np.arange(nx) + 0.5) / nx - 0.5
            y = (np.arange(ny) + 0.5) / ny - 0.5
            z = ((np.arange(nz) - 0.5) * base.dz - 3000.0) / 2000.0
            r = np.sqrt((x / 0.2)[:, None, None] ** 2 + (y / 0.2)[None, :, None] ** 2 + z[None, None, :] ** 2)
            blob = np.where(r < 1.0, 0.5 + 0.5 * np.cos(math.pi * np.minimum(r, 1.0)), 0.0)
            f["qv"] = 1.0e-3 * blob
            f["qc"] = 1.5e-3 * blob * (1.0 + noise(0.2))
            # gradients are taken in a region of steady rain: where rain just begins the fall speed has no derivative
            rain = blob + 0.2 if kind == "adjoint_moist" else blob
            f["qr"] = 1.0e-3 * rain * (1.0 + noise(0.2))
        else:
            for n in ("qc", "qr") + (ICE if kind == "ice" else ()):
                f[n] = f[n] * (1.0 + noise(0.1))
    return base, f


def _workload(base, fields):
    return dataclasses.replace(base, fields=fields)


class _Buffer:
    """A device buffer of the library, for torch.as_tensor, which holds on to
    it: the model that owns the memory lives as long as any tensor over it."""

    def __init__(self, model, ptr, shape, typestr):
        self.owner = model
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3}


class _Views:
    """Tensors over a model's field buffers, one per pointer."""

    def __init__(self, model, case):
        self.m, self.t = model, "<f4" if case["f32"] else "<f8"
        self.shape = (case["nx"], case["ny"], case["nz"])
        self.seen = {}

    def __call__(self, field, slot=0):
        ptr = self.m.device_ptr(field, slot)
        v = self.seen.get(ptr)
        if v is None:
            flat = field in (abi.GA_ACCRAIN, abi.GA_ACCSNOW)
            v = torch.as_tensor(_Buffer(self.m, ptr, self.shape[:2] if flat else self.shape,
                                        "<f8" if flat else self.t), device="cuda")
            self.seen[ptr] = v
        return v


def _model(case, wl, fields):
    prec = abi.GA_PREC_F32 if case["f32"] else abi.GA_PREC_F64
    m = anelastic.Model(_workload(wl, fields), prec, device=0, columns=anelastic.build_columns(wl))
    if case["tuned"]:
        m.tune()
    return m


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        sizes = [(case["nx"], case["ny"], case["nz"])] * case["members"]
        sizes += [(case["nx2"], case["ny2"], case["nz2"])] * case["members2"]
        states = [_state("storm", *s, seed * 1000 + m) for m, s in enumerate(sizes)]
        e = anelastic.Ensemble([b for b, _ in states], abi.GA_PREC_F32)
        for m, (_, f) in enumerate(states):
            e.load_member(m, f)
        if case["tuned"]:
            e.tune()
        return {"case": case, "ensemble": e}
    base, f = _state(kind, case["nx"], case["ny"], case["nz"], seed)
    m = _model(case, base, f)
    s = {"case": case, "model": m, "views": _Views(m, case)}
    if kind.startswith("adjoint"):
        rng = np.random.default_rng(seed + 1)
        for fld in m.lin_fields():  # the sensitivity of a cost function to the final state
            m.lin_set(fld, abi.GA_SLOT_CUR, rng.random(m.n3) - 0.5)
    return s


def _pressure_out(case, dx):
    """Whether a pass hands out the diagnosed pressure too.  It is no part of
    the state, and on wide domains in single precision its longest waves are
    set by the transforms' rounding (1e-4 of it), so it is read in double
    precision or on domains up to 130 km."""
    return not case["f32"] or max(case["nx"], case["ny"]) * dx <= 130.0e3


def run(state):
    case = state["case"]
    if case["kind"] == "ensemble":
        e = state["ensemble"]
        e.step(case["steps"])
        # host access hands out doubles; the members' state is single precision
        return {"%s%d" % (n, m): e.get(m, f).astype(np.float32) for m in range(len(e.members))
                for f, n in enumerate(PROG)}
    m, views = state["model"], state["views"]
    if case["kind"].startswith("adjoint"):
        m.adjoint(case["steps"], case["every"])
        # current and start-of-step slots both hold the initial perturbation: its gradient is their sum
        keep = np.float32 if case["f32"] else np.float64  # host access hands out doubles
        return {PROG[f] + suf: m.lin_get(f, slot).astype(keep, copy=False) for f in m.lin_fields()
                for slot, suf in ((abi.GA_SLOT_CUR, ""), (abi.GA_SLOT_M, "_m"))}
    m.step(case["steps"])
    moist = m.wl.microphysics_option
    out = {}
    for f in range(7 if moist else 4):
        out[PROG[f]] = views(f)
        out[PROG[f] + "_p"] = views(f, abi.GA_SLOT_P)
    if _pressure_out(case, m.wl.dx):
        out["pi"] = views(abi.GA_PI)
    total = torch.float32 if case["f32"] else torch.float64  # totals of increments in the model's precision
    if moist:
        out["accrain"] = views(abi.GA_ACCRAIN).to(total)
    if moist == 2:
        for n, f in abi.ICE_PROG.items():
            out[n] = views(f)
            out[n + "_p"] = views(f, abi.GA_SLOT_P)
        out["accsnow"] = views(abi.GA_ACCSNOW).to(total)
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: per step the state fields read and written once per stage (as
    the three-stage scheme needs them) with the pressure solve's passes; flops:
    faces and tendencies, transforms, vertical solves, point physics."""
    size = 4 if case["f32"] else 8
    kind = case["kind"]

    def step(nx, ny, nz, nf):
        n = nx * ny * nz
        # a stage: nf current and nf start-of-step fields in, nf forecast fields out, the pressure field out
        # and in, the y-transformed half spectrum out and in; then the step's last pass (in, out twice)
        passes = 3 * (3 * nf + 2 + 2) + 3 * nf
        flux = nf * 120 + 60
        fft = 2 * 2.5 * math.log2(max(2, nx * ny)) + 12
        return n * passes * size, n * (3 * (flux + fft) + (150 if nf > 4 else 0))

    if kind == "ensemble":
        parts = [(case["nx"], case["ny"], case["nz"])] * case["members"]
        parts += [(case["nx2"], case["ny2"], case["nz2"])] * case["members2"]
        b = sum(step(*p, 7)[0] for p in parts) * case["steps"] + sum(p[0] * p[1] * p[2] for p in parts) * 7 * 8
        return {"bytes": b, "flops": sum(step(*p, 7)[1] for p in parts) * case["steps"]}
    nf = {"bubble": 4, "jet": 4, "adjoint_dry": 4, "ice": 9}.get(kind, 7)
    b, f = step(case["nx"], case["ny"], case["nz"], nf)
    if kind == "physics":  # diffusion in and out; coefficients, tendencies and their use in each stage
        n = case["nx"] * case["ny"] * case["nz"]
        b += n * size * (14 + 4 * 7)
        f += n * 7 * 100
    if kind.startswith("adjoint"):  # the trajectory twice, and per stage the linearised operators
        b, f = 2 * b + 2 * b, 2 * f + 2 * f
    return {"bytes": b * case["steps"], "flops": f * case["steps"]}


# ---------------------------------------------------------------------------
# the nonlinear step in 64 bits (reference equations: advection.cpp, fluxes.cpp,
# pressure.cpp, boundaries.cpp, kessler.cpp, damping.cpp)
# ---------------------------------------------------------------------------
def _columns(wl):
    nz, dz = wl.nz, wl.dz
    k = np.arange(nz, dtype=np.float64)
    zu, zw = (k - 0.5) * dz, (k - 1.0) * dz
    tb, qb = np.array(wl.fields["tb_in"]), np.array(wl.fields["qb_in"])
    for a in (tb, qb):
        a[0], a[-1] = a[1], a[-2]
    tbv = tb * (1.0 + 0.61 * qb)
    pib = np.zeros(nz)
    pib[1] = (100200.0 / 1.0e5) ** (287.0 / 1004.0) - 9.8 * zu[1] / (1004.0 * tbv[1])
    pib[0] = (100200.0 / 1.0e5) ** (287.0 / 1004.0) + 9.8 * (0 - zu[0]) / (1004.0 * tbv[0])
    for m in range(2, nz):
        pib[m] = pib[m - 1] - 9.8 * (zu[m] - zu[m - 1]) / (1004.0 * 0.5 * (tbv[m] + tbv[m - 1]))
    rhou = 1.0e5 * pib ** (717.0 / 287.0) / (287.0 * tbv)
    rhow = np.zeros(nz)
    rhow[1:] = 0.5 * (rhou[1:] + rhou[:-1])
    rhow[0] = rhow[1]
    tbv[0], tbv[-1] = tbv[1], tbv[-2]
    lat = -89.462997 + wl.corner_lat + wl.dx / 111000.0 * (1.0 + np.arange(wl.ny))
    cor = 2 * 7.292e-5 * np.sin(lat * math.pi / 180.0)
    ray = np.zeros((2, nz))
    r = wl.rayleigh_damping_z
    for m, z in enumerate((zu, zw)):
        ray[m, r:] = 0.025 * (1.0 - np.cos(math.pi * (z[r:] - zu[r]) / (z[-1] - zu[r])))
    return {"tb": tb, "qb": qb, "tbv": tbv, "rhou": rhou, "rhow": rhow, "f": cor, "ray_u": ray[0], "ray_w": ray[1]}


class _Exact:
    """The RK3 step on FP64 tensors with the three rotation buffers: a
    non-periodic domain on a uniform vertical grid, dry or with Kessler
    microphysics and Eulerian rain."""

    def __init__(self, wl, fields):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        as_t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)  # noqa: E731
        self.wl, self.dev = wl, dev
        self.c = {k: as_t(v) for k, v in _columns(wl).items()}
        self.bar = {n: as_t(fields[n]) for n in abi.BAR_NAMES}
        self.names = PROG if wl.microphysics_option else PROG[:4]
        self.cur = {n: as_t(fields[n]) for n in self.names}
        self.M = {n: v.clone() for n, v in self.cur.items()}
        self.P = {n: torch.zeros_like(v) for n, v in self.cur.items()}
        self.pi = torch.zeros(wl.nx, wl.ny, wl.nz, dtype=torch.float64, device=dev)
        self.vt = torch.zeros_like(self.pi)
        self.accrain = torch.zeros(wl.nx, wl.ny, dtype=torch.float64, device=dev)
        self._sponge()
        self._spectral()

    def _sponge(self):
        wl = self.wl
        nx, ny = wl.nx, wl.ny
        g = torch.ones(nx, ny, dtype=torch.float64, device=self.dev)
        lo = lambda n: 0.5 * (np.cos(math.pi * np.arange(n) / max(n, 1)) + 1.0)  # noqa: E731
        hi = lambda n: 0.5 * (np.cos(math.pi * ((np.arange(n) + 1) / max(n, 1) - 1.0)) + 1.0)  # noqa: E731
        for i, v in zip(range(nx - wl.boundary_width_east, nx), hi(wl.boundary_width_east)):
            g[i, 1:] *= 1.0 - v
        for i, v in enumerate(lo(wl.boundary_width_west)):
            g[i, 1:] *= 1.0 - v
        for j, v in enumerate(lo(wl.boundary_width_south)):
            g[1:, j] *= 1.0 - v
        for j, v in zip(range(ny - wl.boundary_width_north, ny), hi(wl.boundary_width_north)):
            g[1:, j] *= 1.0 - v
        self.sponge = g[:, :, None]

    def _spectral(self):
        wl, c = self.wl, self.c
        kx = 2 * math.pi * torch.arange(wl.nx, dtype=torch.float64, device=self.dev) / wl.nx
        ky = 2 * math.pi * torch.arange(wl.ny // 2 + 1, dtype=torch.float64, device=self.dev) / wl.ny
        self.h = torch.cos(kx)[:, None] + torch.cos(ky)[None, :] - 2.0
        self.a = c["rhow"] / wl.dz ** 2  # lower coefficient at k, upper at k is a[k+1]

    @staticmethod
    def _up(x):
        return torch.where(x > 0, 1.0, -1.0).to(x.dtype)

    @staticmethod
    def _five(s, sign):
        m2, m1, z, p1, p2, p3 = s
        c6 = 37.0 / 60.0 * (p1 + z) - 2.0 / 15.0 * (p2 + m1) + (p3 + m2) / 60.0
        return c6 + sign / 60.0 * (-(p3 - m2) + 5.0 * (p2 - m1) - 10.0 * (p1 - z))

    def _east(self, a, sign):
        n = self.wl.nx - 5
        return self._five([a[m:m + n, 3:-3] for m in range(6)], sign)

    def _north(self, a, sign):
        n = self.wl.ny - 5
        return self._five([a[3:-3, m:m + n] for m in range(6)], sign)

    def _top(self, a, sign):
        """Faces between k and k+1 for k = 1..nz-2 of the advected columns."""
        a = a[3:-3, 3:-3]
        f = 0.5 * (a[..., 2:] + a[..., 1:-1])
        m1, z, p1, p2 = a[..., 1:-3], a[..., 2:-2], a[..., 3:-1], a[..., 4:]
        inner = 7.0 / 12.0 * (p1 + z) - (p2 + m1) / 12.0 + sign[..., 1:-1] / 12.0 * ((p2 - m1) - 3.0 * (p1 - z))
        return torch.cat([f[..., :1], inner, f[..., -1:]], -1)

    def _flux(self, s, b, adv, advb, along):
        """Face flux of field s (basic state b or None) along one direction."""
        tot = advb + adv
        f = along(s, self._up(tot)) * tot
        return f if b is None else f + adv * along(b, self._up(adv))

    def _tend(self, e, n, t, bottom=None):
        wl, c = self.wl, self.c
        zero = torch.zeros_like(t[..., :1]) if bottom is None else bottom
        t = torch.cat([zero, t], -1)  # faces k = 0..nz-2
        rw = c["rhow"]
        div = -(wl.dt / wl.dx) * (e[1:] - e[:-1])[..., 1:-1] - (wl.dt / wl.dx) * (n[:, 1:] - n[:, :-1])[..., 1:-1]
        return div - (wl.dt / wl.dz) * (rw[2:] * t[..., 1:] - rw[1:-1] * t[..., :-1]) / c["rhou"][1:-1]

    def _fall(self, q):
        c = self.c
        v = 36.34 * torch.clamp(q * 0.001 * c["rhou"], min=0.0) ** 0.1364 * torch.sqrt(c["rhou"][1] / c["rhou"])
        v = torch.where(q > 1e-12, v, torch.zeros_like(v))
        v[..., 0] = v[..., 1]
        v[..., -1] = self.vt[..., -1]
        return v

    def _advect(self, st):
        wl, c, C, B = self.wl, self.c, self.cur, self.bar
        U, V, Wf = C["u"], C["v"], C["w"]
        ii, jj, kk = slice(3, -3), slice(3, -3), slice(1, -1)
        pair_e = lambda a: 0.5 * (a[3:-2, 3:-3] + a[2:-3, 3:-3])  # noqa: E731
        pair_n = lambda a: 0.5 * (a[3:-3, 3:-2] + a[3:-3, 2:-3])  # noqa: E731
        cor = c["f"][3:-3, None]
        new = {}
        # u
        e = self._flux(U, B["ubar"], pair_e(U), pair_e(B["ubar"]), self._east)
        av = lambda a: 0.5 * (a[3:-3, 3:-2] + a[2:-4, 3:-2])  # noqa: E731
        n = self._flux(U, B["ubar"], av(V), av(B["vbar"]), self._north)
        aw = lambda a: 0.5 * (a[3:-3, 3:-3, 2:] + a[2:-4, 3:-3, 2:])  # noqa: E731
        t = self._flux(U, B["ubar"], aw(Wf), aw(B["wbar"]), self._top)
        over = 0.25 * (V[3:-3, 3:-3] + V[3:-3, 4:-2] + V[2:-4, 3:-3] + V[2:-4, 4:-2])[..., kk]
        new["u"] = self._tend(e, n, t) + wl.dt * cor * over
        # v
        au = lambda a: 0.5 * (a[3:-2, 3:-3] + a[3:-2, 2:-4])  # noqa: E731
        e = self._flux(V, B["vbar"], au(U), au(B["ubar"]), self._east)
        n = self._flux(V, B["vbar"], pair_n(V), pair_n(B["vbar"]), self._north)
        aw = lambda a: 0.5 * (a[3:-3, 3:-3, 2:] + a[3:-3, 2:-4, 2:])  # noqa: E731
        t = self._flux(V, B["vbar"], aw(Wf), aw(B["wbar"]), self._top)
        over = 0.25 * (U[3:-3, 3:-3] + U[4:-2, 3:-3] + U[3:-3, 2:-4] + U[4:-2, 2:-4])[..., kk]
        new["v"] = self._tend(e, n, t) - wl.dt * cor * over
        # scalars
        ue, ube = U[3:-2, 3:-3], B["ubar"][3:-2, 3:-3]
        vn, vbn = V[3:-3, 3:-2], B["vbar"][3:-3, 3:-2]
        wt, wbt = Wf[3:-3, 3:-3, 2:], B["wbar"][3:-3, 3:-3, 2:]
        for name in self.names[3:]:
            s, b = C[name], {"th": B["thbar"], "qv": B["qbar"]}.get(name)
            base = {"th": c["tb"], "qv": c["qb"]}.get(name)
            e = self._flux(s, b, ue, ube, self._east)
            n = self._flux(s, b, vn, vbn, self._north)
            if name != "qr":
                tend = self._tend(e, n, self._flux(s, b, wt, wbt, self._top))
            else:
                vt = self._fall(s)[3:-3, 3:-3]
                wf = wbt + wt - 0.5 * (vt[..., 1:-1] + vt[..., 2:])
                bot = -0.5 * (vt[..., 1:2] + vt[..., :1]) * 0.5 * (s[3:-3, 3:-3, :1] + s[3:-3, 3:-3, 1:2])
                tend = self._tend(e, n, self._top(s, self._up(wf)) * wf, bot)
                self.vt[ii, jj, :-1] = vt[..., :-1]
            if base is not None:
                w = Wf[3:-3, 3:-3]
                zab = 0.5 * (c["rhow"][2:] * w[..., 2:] * (base[2:] - base[1:-1])
                             + c["rhow"][1:-1] * w[..., 1:-1] * (base[1:-1] - base[:-2])) / c["rhou"][1:-1]
                tend = tend - (wl.dt / wl.dz) * zab
            new[name] = tend
        buoy = C["th"] / c["tbv"]
        if len(self.names) > 4:
            buoy = buoy + 0.61 * C["qv"] - C["qc"] - C["qr"]
        buoy = buoy[3:-3, 3:-3]
        for name, tend in new.items():
            self.P[name][ii, jj, kk] = self.M[name][ii, jj, kk] + st * tend
        self.P["w"][ii, jj, 2:-1] = self.M["w"][ii, jj, 2:-1] + st * wl.dt * 9.8 * 0.5 * (
            buoy[..., 2:-1] + buoy[..., 1:-2])

    def _solve(self, st):
        wl, c = self.wl, self.c
        nx, ny, nz = wl.nx, wl.ny, wl.nz
        for n in ("u", "v", "w"):
            a = self.P[n][:, :, 1:-1]
            a[0, 1:-1], a[-1, 1:-1] = a[1, 1:-1].clone(), a[-2, 1:-1].clone()
            a[:, 0], a[:, -1] = a[:, 1].clone(), a[:, -2].clone()
        u, v, w = (self.P[n] for n in ("u", "v", "w"))
        d = c["rhou"][1:-1] * ((u[2:, 1:-1] - u[1:-1, 1:-1]) / wl.dx + (v[1:-1, 2:] - v[1:-1, 1:-1]) / wl.dx)[..., 1:-1]
        d = d + (c["rhow"][2:] * w[1:-1, 1:-1, 2:] - c["rhow"][1:-1] * w[1:-1, 1:-1, 1:-1]) / wl.dz
        d = d / (st * wl.dt)
        d = torch.cat([d[:1], d, d[-1:]], 0)
        d = torch.cat([d[:, :1], d, d[:, -1:]], 1)
        x = torch.fft.rfft2(d, dim=(0, 1)).permute(2, 0, 1).contiguous()  # levels 1..nz-2
        a, nl = self.a, nz - 2
        gam, den = [], None
        for r in range(nl):  # tridiagonal elimination, all wavenumbers at once
            k = r + 1
            low = 0.0 if r == 0 else a[k]
            upper = 0.0 if r == nl - 1 else a[k + 1]
            b = c["rhou"][k] * 2.0 * self.h / wl.dx ** 2 - (low + upper)
            den = 1.0 / (b if r == 0 else b - low * gam[-1])
            gam.append(upper * den)
            x[r] = (x[r] if r == 0 else x[r] - low * x[r - 1]) * den
        x[nl - 1, 0, 0] = 0.0  # the mean mode's gauge
        for r in range(nl - 2, -1, -1):
            x[r] -= gam[r] * x[r + 1]
        p = torch.fft.irfft2(x, s=(nx, ny), dim=(1, 2)).permute(1, 2, 0)
        self.pi[:, :, 0], self.pi[:, :, -1] = p[..., 0], p[..., -1]
        inner = p[1:-1, 1:-1]
        inner = torch.cat([inner[:1], inner, inner[-1:]], 0)
        self.pi[:, :, 1:-1] = torch.cat([inner[:, :1], inner, inner[:, -1:]], 1)

    def _project(self, st):
        wl, P, p = self.wl, self.P, self.pi
        q = (slice(1, -1), slice(1, -1), slice(1, -1))
        P["u"][q] -= st * wl.dt / wl.dx * (p[1:-1, 1:-1] - p[:-2, 1:-1])[..., 1:-1]
        P["v"][q] -= st * wl.dt / wl.dx * (p[1:-1, 1:-1] - p[1:-1, :-2])[..., 1:-1]
        P["w"][1:-1, 1:-1, 2:-1] -= st * wl.dt / wl.dz * (p[1:-1, 1:-1, 2:-1] - p[1:-1, 1:-1, 1:-2])

    def _clip(self):
        if len(self.names) > 4:
            P, c = self.P, self.c
            P["qc"].clamp_(min=0.0)
            P["qr"].clamp_(min=0.0)
            q = (slice(1, -1), slice(1, -1), slice(1, -1))
            P["qv"][q] = torch.maximum(P["qv"][q], -(self.bar["qbar"] + c["qb"])[q])

    def _bounds(self, rayleigh=False):
        for n in self.names:
            a = self.P[n]
            a[:, :, 1:] *= self.sponge
            if n == "w":
                a[1:, 1:, 0] = a[1:, 1:, 1] = a[1:, 1:, -1] = 0.0
            else:
                a[1:, 1:, 0], a[1:, 1:, -1] = a[1:, 1:, 1], a[1:, 1:, -2]
            if rayleigh and n in PROG[:4]:
                a[1:-1, 1:-1] *= 1.0 - (self.c["ray_w"] if n == "w" else self.c["ray_u"])

    def _kessler(self):
        wl, c, P, q = self.wl, self.c, self.P, (slice(1, -1), slice(1, -1), slice(1, -1))
        cp, lv = 1004.0, 2.5e6
        th, qv, qc, qr = (P[n][q] for n in ("th", "qv", "qc", "qr"))
        thb = (self.bar["thbar"] + c["tb"])[q]
        qvb = (self.bar["qbar"] + c["qb"])[q]
        rho = c["rhou"][1:-1]
        press = (self.pi / (cp * c["tbv"]) + self.bar["pbar"])[q]
        pd = 1.0e5 * press ** (cp / 287.0)
        z = torch.zeros_like(th)

        def sat(t):
            es = 611.2 * torch.exp(17.67 * (t - 273.15) / (t - 29.65))
            return es, 0.62197 * es / (pd - es)

        rain = qr > 1e-12
        qp = torch.where(rain, qr, z)
        auto = torch.where(qc > 1e-3, 0.001 * (qc - 1e-3) * wl.dt, z)
        accr = rho * 2.2 * qc * qp ** 0.875 * wl.dt
        _, qs = sat((th + thb) * press)
        vent = 1.6 + 30.3922 * (rho * qp) ** 0.2046
        ev = (1.0 - (qv + qvb) / qs) * vent * (rho * qp) ** 0.525 / (2.03e4 + 9.58e6 / (pd * qs)) / rho * wl.dt
        ev = torch.where(rain, torch.clamp(torch.minimum(qr, ev), min=0.0), z)
        conv = torch.minimum(auto + accr, qc)
        qv, qc, qr = qv + ev, qc - conv, qr + (conv - ev)
        th = th - lv / (cp * press) * ev
        t = (th + thb) * press
        es, qs = sat(t)
        phi = pd / (pd - es) * qs * (17.67 * (273.15 - 29.65) * lv / cp) / (t - 29.65) ** 2
        vap = qv + qvb
        cond = torch.where(vap > qs, (vap - qs) / (1.0 + phi),
                           torch.where((vap < qs) & (qc > 0), -torch.minimum(qc, (qs - vap) / (1.0 + phi)), z))
        P["th"][q], P["qv"][q] = th + lv / (cp * press) * cond, qv - cond
        P["qc"][q], P["qr"][q] = qc + cond, qr
        fall = c["rhow"][1] * 0.5 * (self.vt[1:-1, 1:-1, 0] + self.vt[1:-1, 1:-1, 1])
        self.accrain[1:-1, 1:-1] += fall * 0.5 * (P["qr"][1:-1, 1:-1, 0] + P["qr"][1:-1, 1:-1, 1]) * wl.dt

    def step(self):
        for s, st in enumerate((1.0 / 3.0, 0.5, 1.0)):
            self._advect(st)
            self._solve(st)
            self._project(st)
            self._clip()
            self._bounds()
            if s < 2:
                self.cur, self.P = self.P, self.cur
        if len(self.names) > 4:
            self._kessler()
        self._bounds(rayleigh=True)
        self.M = {n: v.clone() for n, v in self.P.items()}
        self.cur, self.P = self.P, self.cur


def exact(case, seed):
    """The step in 64 bits, for the kinds it covers; none for the ice scheme,
    the hydrostatic set, turbulence and diffusion, semi-Lagrangian rain, and
    the linearisations."""
    kind = case["kind"]
    if kind not in ("bubble", "storm", "jet", "squall", "ensemble"):
        return None
    if kind == "ensemble":
        sizes = [(case["nx"], case["ny"], case["nz"])] * case["members"]
        sizes += [(case["nx2"], case["ny2"], case["nz2"])] * case["members2"]
        if case["steps"] * sum(a * b * c for a, b, c in sizes) > 2e8:
            return None
        out = {}
        for m, s in enumerate(sizes):
            x = _Exact(*_state("storm", *s, seed * 1000 + m))
            for _ in range(case["steps"]):
                x.step()
            out.update({"%s%d" % (n, m): x.cur[n].reshape(-1).cpu().numpy() for n in x.names})
        return out
    x = _Exact(*_state(kind, case["nx"], case["ny"], case["nz"], seed))
    for _ in range(case["steps"]):
        x.step()
    out = {}
    for n in x.names:
        out[n], out[n + "_p"] = x.cur[n], x.P[n]
    if _pressure_out(case, x.wl.dx):
        out["pi"] = x.pi
    if len(x.names) > 4:
        out["accrain"] = x.accrain
    return out
