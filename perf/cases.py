"""The work that users of the groundwater step have it do, as measurable cases.

Every case is one scenario through the public entry points: (re)initialise the
domain, take a few adaptive steps the way the driver loop does, read back head
and moisture.  ``listed()`` gives fixed cases over the range of domains this
repository configures, tests and benchmarks; ``draw(rng)`` more of the same
ranges.  ``exact(case, seed)`` is a plain float64 torch restatement of the
groundwater-only step with its linear systems solved to rounding.
"""
import ctypes
import math

import numpy as np
import torch

from frehg_b200.batch import RichardsBatch
from frehg_b200.config import (IC_FORMS, BoundaryCondition, Domain, Groundwater, GwConfig,
                               InitialCondition, Solver, SoilType, Timestep, whole_footprint)
from frehg_b200.coupling import Coupler
from frehg_b200.gw import RichardsSolver, _check

_dp = ctypes.POINTER(ctypes.c_double)

# Residual target of the mixed and FP64-line solves on the hillslopes.  The
# post-allocation branches on the solved head, so a run's fields are as
# reproducible as its solves: at the default 3e-12 the head after ten steps of
# a hillslope is 1e-9 from that of another equally good solve, at 1e-13 2e-11.
TIGHT = 1.0e-13

# Largest domain (cells) for which exact() is computed: about 10 s of plain
# torch, most of it point-Jacobi CG on the cold first step.
EXACT_CELLS = 9_000_000


def _box(name, nx, ny, nz, precision, steps):
    return {"name": name, "kind": "box", "nx": nx, "ny": ny, "nz": nz, "precision": precision,
            "steps": steps}


def _hill(name, nx, ny, nz, precision, dt0, steps):
    return {"name": name, "kind": "hill", "nx": nx, "ny": ny, "nz": nz, "precision": precision,
            "dt0": dt0, "steps": steps}


def _ensemble(name, members, most, deepest, precision, steps):
    return {"name": name, "kind": "ensemble", "members": members, "most": most,
            "deepest": deepest, "precision": precision, "steps": steps}


def _coupled(name, nx, ny, nz, precision, windows):
    return {"name": name, "kind": "coupled", "nx": nx, "ny": ny, "nz": nz,
            "precision": precision, "windows": windows}


def listed():
    return [
        # The smallest call: a plot-scale box (the smoke run's), all latency.
        _box("box_8x6x20_fp64", 8, 6, 20, "fp64", 20),
        # Infiltration into the 32x32x50 box: the reference-CPU-runnable case.
        _box("box_32x32x50_fp64", 32, 32, 50, "fp64", 20),
        _box("box_32x32x50_mixed", 32, 32, 50, "mixed", 20),
        # Deep columns (more than 256 layers): the mixed form's tiled line solve.
        _box("box_24x20x300_mixed", 24, 20, 300, "mixed", 10),
        # A hillslope plot of the benchmark slab's construction, the default form.
        _hill("hill_64x64x128_fp64", 64, 64, 128, "fp64", 60.0, 4),
        # The same in the mixed form, as production runs take it.
        _hill("hill_64x64x128_mixed", 64, 64, 128, "mixed", 60.0, 12),
        # Ragged domains: no extent a multiple of anything.
        _hill("hill_97x61x75_fp64_line", 97, 61, 75, "fp64_line", 60.0, 8),
        _hill("hill_131x113x127_fp64", 131, 113, 127, "fp64", 60.0, 3),
        # A catchment tile, larger than L2, in the headline form.
        _hill("hill_256x256x128_mixed", 256, 256, 128, "mixed", 60.0, 20),
        # The benchmark slab, in the reference's own solver form.
        _hill("hill_512x512x128_fp64", 512, 512, 128, "fp64", 0.5, 2),
        # A calibration ensemble of uneven boxes stepped as one batch.
        _ensemble("ensemble_24_mixed", 24, 128, 200, "mixed", 12),
        # Coupled surface water: a V-catchment of the reference's benchmark
        # size, lockstep windows of its dt = 2 s.
        _coupled("coupled_101x55x25_fp64", 101, 55, 25, "fp64", 12),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["box", "box", "hill", "hill", "hill", "ensemble", "coupled"])
    if kind == "box":
        precision = rng.choice(["fp64", "fp64", "mixed", "mixed", "fp64_line"])
        deepest = 256 if precision == "fp64_line" else 320
        c = _box("", _log(rng, 6, 96), _log(rng, 6, 96), _log(rng, 16, deepest), precision,
                 rng.randint(8, 20))
    elif kind == "hill":
        precision = rng.choice(["fp64", "fp64", "mixed", "mixed", "mixed", "fp64_line"])
        c = _hill("", _log(rng, 40, 260), _log(rng, 40, 260), rng.randint(60, 160), precision,
                  60.0, rng.randint(2, 4) if precision == "fp64" else rng.randint(6, 12))
    elif kind == "ensemble":
        c = _ensemble("", rng.randint(8, 24), rng.randint(48, 128), rng.randint(64, 200),
                      rng.choice(["fp64", "mixed"]), rng.randint(6, 12))
    else:
        c = _coupled("", _log(rng, 20, 120), _log(rng, 20, 120), rng.randint(12, 40),
                     rng.choice(["fp64", "fp64", "mixed"]), rng.randint(8, 16))
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _smooth(shape, corr, gen):
    """Zero-mean, unit-variance Gaussian field of correlation length `corr` cells."""
    noise = torch.randn(shape, generator=gen, device=gen.device, dtype=torch.float64)
    spec = torch.fft.rfftn(noise)
    freqs = [torch.fft.fftfreq(n, device=gen.device, dtype=torch.float64) for n in shape[:-1]]
    freqs.append(torch.fft.rfftfreq(shape[-1], device=gen.device, dtype=torch.float64))
    for axis, f in enumerate(freqs):
        filt = torch.exp(-((math.pi * corr * f) ** 2))
        spec *= filt.reshape([-1 if a == axis else 1 for a in range(len(shape))])
    field = torch.fft.irfftn(spec, s=shape)
    field -= field.mean()
    return field / field.std()


def _uniform(shape, lo, hi, gen):
    return torch.rand(shape, generator=gen, device=gen.device, dtype=torch.float64) * (hi - lo) + lo


def _box_config(nx, ny, nz, precision, rng, dt0=10.0, coin=False):
    """A homogeneous box of the ensemble's soils: ponded head on top (with
    `coin`, or a flux by a fair draw), free drainage below, closed sides."""
    ks = float(np.exp(np.log(1e-5) + 0.5 * rng.standard_normal()))
    soil = SoilType("box", ks, ks, ks, 0.40, 0.05, float(rng.uniform(0.5, 3.0)),
                    float(rng.uniform(1.4, 2.5)), 0.0)
    h0 = float(rng.uniform(-3.0, -0.2))
    ponded = bool(rng.integers(0, 2)) if coin else True
    fp = whole_footprint(nx, ny)
    top = (BoundaryCondition("ponded-top", fp, "groundwater_top", "head", "constant", 0.01)
           if ponded else
           BoundaryCondition("recharge-top", fp, "groundwater_top", "flux", "constant", -1e-6))
    return GwConfig(
        domain=Domain(nx=nx, ny=ny, nz=nz, dx=1.0, dy=1.0, dz=0.02, bottom_elevation=0.0),
        soil_types=[soil],
        groundwater=Groundwater(timestep=Timestep(dt_init=dt0, dt_min=1e-3, dt_max=600.0),
                                specific_storage=1e-5),
        initial=InitialCondition("head", h0),
        solver=Solver(precision=precision, max_iterations=20000),
        boundary_conditions=[top, BoundaryCondition("free-drainage", fp, "groundwater_bottom",
                                                    "flux", "gravity")])


def _hill_config(case, seed):
    """The benchmark slab's construction at the case's size: sloping bed with
    bumps, per-cell heterogeneous soil, water table 2 m down, recharge on top."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=_device()).manual_seed(seed)
    X, Y = np.meshgrid(np.arange(nx) + 0.5, np.arange(ny) + 0.5)
    bath = -0.02 * X
    for _ in range(max(1, nx * ny // 4096)):
        cx, cy = rng.uniform(0, nx), rng.uniform(0, ny)
        bath += 0.5 * np.exp(-((X - cx) ** 2 + (Y - cy) ** 2) / (2.0 * 16.0 ** 2))
    shape = (ny, nx, nz)
    ks = torch.exp(math.log(1e-5) + _smooth(shape, 8.0, gen)).cpu().numpy()
    soil = dict(ksx=ks, ksy=ks, ksz=ks, vg_alpha=_uniform(shape, 0.5, 3.0, gen).cpu().numpy(),
                vg_n=_uniform(shape, 1.4, 2.5, gen).cpu().numpy())
    fp = whole_footprint(nx, ny)
    return GwConfig(
        domain=Domain(nx=nx, ny=ny, nz=nz, dx=1.0, dy=1.0, dz=0.05, bottom_elevation=bath,
                      follow_terrain=True, terrain_layers="uniform"),
        soil_types=[SoilType("s", 0, 0, 0, 0.40, 0.05, 0, 0, 0.0)],
        groundwater=Groundwater(timestep=Timestep(dt_init=case["dt0"], dt_min=1e-3, dt_max=600.0),
                                specific_storage=1e-5),
        initial=InitialCondition("water_table", bath - 2.0),
        solver=Solver(precision=case["precision"], max_iterations=20000, outer_rtol=TIGHT),
        boundary_conditions=[
            BoundaryCondition("recharge", fp, "groundwater_top", "flux", "constant", -1e-6),
            BoundaryCondition("free-drainage", fp, "groundwater_bottom", "flux", "gravity")],
        cell_soil=soil)


def _coupled_config(case, seed):
    """A V-catchment: two planes falling to a channel that falls to the outlet,
    heterogeneous soil, closed sides and bottom, shallow water table."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    rng = np.random.default_rng(seed)
    X, Y = np.meshgrid(np.arange(nx) + 0.5, np.arange(ny) + 0.5)
    bath = -(0.02 * Y + 0.05 * (nx / 2 - np.abs(X - nx / 2)))
    ks = 1e-5 * np.exp(0.5 * rng.standard_normal((ny, nx, nz)))
    cfg = GwConfig(
        domain=Domain(nx=nx, ny=ny, nz=nz, dx=1.0, dy=1.0, dz=0.1, bottom_elevation=bath,
                      follow_terrain=True, terrain_layers="uniform"),
        soil_types=[SoilType("loam", 1e-5, 1e-5, 1e-5, 0.45, 0.08, 2.0, 1.8, 0.0)],
        groundwater=Groundwater(timestep=Timestep(dt_init=2.0, dt_min=1e-2, dt_max=60.0),
                                specific_storage=1e-5),
        initial=InitialCondition("water_table", bath - 0.5),
        solver=Solver(precision=case["precision"], max_iterations=20000, outer_rtol=TIGHT),
        cell_soil=dict(ksx=ks, ksy=ks, ksz=ks))
    # The channel holds 5 cm of water; rain falls on the whole catchment.
    pond = np.where(np.abs(X - nx / 2) < 2.0, 0.05, 0.0)
    rain = rng.uniform(1e-4, 3e-4, size=(ny, nx))
    return cfg, bath, pond, rain


def _member_configs(case, seed):
    rng = np.random.default_rng(seed)
    cfgs = []
    # The sizes are the case's own, drawn alike for every seed: the same work.
    sizes = np.random.default_rng(case["members"] * 1000 + case["most"])
    for _ in range(case["members"]):
        nx, ny = (int(sizes.integers(16, case["most"] + 1)) for _ in range(2))
        nz = int(sizes.integers(32, case["deepest"] + 1))
        cfgs.append(_box_config(nx, ny, nz, case["precision"], rng, coin=True))
    return cfgs


def _halo(a):
    return np.pad(a, 1, mode="edge")


def prepare(case, seed):
    if case["kind"] == "ensemble":
        members = [RichardsSolver(c) for c in _member_configs(case, seed)]
        return {"case": case, "members": members, "batch": RichardsBatch(members)}
    if case["kind"] == "coupled":
        cfg, bath, pond, rain = _coupled_config(case, seed)
        s = RichardsSolver(cfg)
        s.attachCoupling(min_depth=1e-3)
        bed = _halo(bath) + s.elevationOffset()
        s.setSurface("bottom", bed)
        return {"case": case, "solver": s, "coupler": Coupler(s, sync=True, dt=2.0, dt_init=2.0),
                "bed": bed, "pond": _halo(pond), "rain": _halo(rain)}
    if case["kind"] == "box":
        cfg = _box_config(case["nx"], case["ny"], case["nz"], case["precision"],
                          np.random.default_rng(seed))
    else:
        cfg = _hill_config(case, seed)
    return {"case": case, "solver": RichardsSolver(cfg)}


# ------------------------------------------------------------------ passes
def _reinitialise(s):
    """The domain back at its initial condition, for the next scenario."""
    ic = s.cfg.initial
    if np.isscalar(ic.value):
        rc = s.lib.frehg_gw_init_state(s.h, IC_FORMS[ic.form], float(ic.value), None)
    else:
        rc = s.lib.frehg_gw_init_state(s.h, IC_FORMS[ic.form], 0.0,
                                       np.ascontiguousarray(ic.value).ctypes.data_as(_dp))
    _check(s.lib, rc)
    s.t = 0.0


def _run_coupled(state):
    s, cp, bed = state["solver"], state["coupler"], state["bed"]
    _reinitialise(s)
    cp.restore(0.0, 2.0, 0.0)
    for name in ("seep_accum", "gain", "bounce", "qss"):
        s.setSurface(name, 0.0)
    eta = bed + state["pond"]
    t = 0.0
    for _ in range(state["case"]["windows"]):
        t += 2.0
        eta = eta + 2.0 * state["rain"]
        depth = eta - bed
        depth[depth <= 1e-3] = 0.0
        s.setSurface("eta", eta)
        s.setSurface("dept", depth)
        cp.step(t, 2.0)
        eta = s.surface("eta")
    return {"h": s.head(), "wc": s.waterContent(), "eta": eta[1:-1, 1:-1],
            "seep": s.surface("seep_accum")[1:-1, 1:-1]}


def run(state):
    case = state["case"]
    if case["kind"] == "coupled":
        return _run_coupled(state)
    if case["kind"] == "ensemble":
        for i, s in enumerate(state["members"]):
            _reinitialise(s)
            state["batch"].set_dt(i, s.cfg.groundwater.timestep.dt_init)
        for _ in range(case["steps"]):
            state["batch"].step()
        return [{"h": s.head(), "wc": s.waterContent()} for s in state["members"]]
    s = state["solver"]
    _reinitialise(s)
    dt = s.cfg.groundwater.timestep.dt_init
    for _ in range(case["steps"]):
        s.t += dt
        s.step(s.t, dt)
        dt = s.nextDt()
    return {"h": s.head(), "wc": s.waterContent()}


def work(case):
    """What one pass cannot do without.  Per cell and step: the state (head
    and moisture) read and written, the per-cell soil and mesh arrays read
    once; at the end head and moisture read out.  Operations: the retention
    and conductivity curves (about 400 per cell and step)."""
    steps = case["windows"] if case["kind"] == "coupled" else case["steps"]
    if case["kind"] == "ensemble":
        cells = sum(c.domain.nx * c.domain.ny * c.domain.nz for c in _member_configs(case, 0))
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
    words = {"box": 4, "ensemble": 4, "hill": 4 + 3 + 8, "coupled": 4 + 1 + 8}[case["kind"]]
    return {"bytes": 8.0 * cells * (steps * words + 2), "flops": 400.0 * cells * steps}


# ------------------------------------------------------------------ 64-bit restatement
def exact(case, seed):
    if case["kind"] == "coupled":
        return None  # the coupled top has no compact plain form
    if case["kind"] == "ensemble":
        return [_exact_run(c, case["steps"]) for c in _member_configs(case, seed)]
    if case["nx"] * case["ny"] * case["nz"] > EXACT_CELLS:
        return None
    cfg = (_hill_config(case, seed) if case["kind"] == "hill" else
           _box_config(case["nx"], case["ny"], case["nz"], case["precision"],
                       np.random.default_rng(seed)))
    return _exact_run(cfg, case["steps"])


def _shift(a, axis, by):
    """a's neighbour along `axis` (index + by), zero outside the domain."""
    out = torch.zeros_like(a)
    n = a.shape[axis]
    if by > 0:
        out.narrow(axis, 0, n - by).copy_(a.narrow(axis, by, n - by))
    else:
        out.narrow(axis, -by, n + by).copy_(a.narrow(axis, 0, n + by))
    return out


class _Soil:
    def __init__(self, cfg, shape, dev):
        t = cfg.soil_types[0]

        def field(name, value):
            v = (cfg.cell_soil or {}).get(name, value)
            return torch.as_tensor(v, dtype=torch.float64, device=dev).expand(shape)

        self.kx, self.kz = field("ksx", t.ksx), field("ksz", t.ksz)
        self.a, self.n = field("vg_alpha", t.vg_alpha), field("vg_n", t.vg_n)
        self.ts, self.tr, self.aev = t.theta_s, t.theta_r, t.aev
        self.m = 1.0 - 1.0 / self.n

    def se(self, h):
        return (1.0 + (self.a * h).abs() ** self.n) ** -self.m

    def theta(self, h):
        wc = torch.where(h > self.aev, torch.full_like(h, self.ts),
                         self.tr + (self.ts - self.tr) * self.se(h))
        return wc.clamp(self.tr, self.ts)

    def head(self, wc):
        wc = wc.clamp(min=self.tr + 1e-7)
        ratio = (self.ts - self.tr) / (wc - self.tr)
        h = -(1.0 / self.a) * (ratio ** (1.0 / self.m) - 1.0).clamp(min=0.0) ** (1.0 / self.n)
        return torch.where(wc < self.ts, h, torch.zeros_like(h))

    def capacity(self, h):
        ah = (self.a * h).abs()
        c = (self.a * self.n * self.m * (self.ts - self.tr) * ah ** (self.n - 1.0) /
             (1.0 + ah ** self.n) ** (self.m + 1.0))
        return torch.where(h > 0.0, torch.zeros_like(h), c)

    def conductivity(self, h, ks):
        se = self.se(h)
        br = 1.0 - (1.0 - se ** (1.0 / self.m)).clamp(min=0.0) ** self.m
        return torch.where(h > 0.0, ks, torch.minimum(ks * se.sqrt() * br * br, ks))

    def dk_dtheta(self, wc):
        wc = torch.where((wc > 0.9999 * self.ts) & (wc < self.ts),
                         torch.full_like(wc, 0.9999 * self.ts), wc)
        se = (wc - self.tr) / (self.ts - self.tr)
        base = 1.0 - se ** (1.0 / self.m)
        t0 = base ** self.m
        t1 = 0.5 * self.kz * se ** -0.5 * (1.0 - t0) ** 2
        t2 = (2.0 * self.kz * se ** ((2.0 - self.m) / (2.0 * self.m)) * (1.0 - t0) *
              base ** (self.m - 1.0))
        return (t1 + t2) / (self.ts - self.tr)


def _exact_run(cfg, steps):
    """Head and moisture after `steps` adaptive steps of a groundwater-only
    domain with closed sides, a head or flux top and a freely draining bottom
    (consistent predictor-corrector, arithmetic faces, surplus dropped)."""
    dev = _device()
    d, g = cfg.domain, cfg.groundwater
    ny, nx, nz, dz = d.ny, d.nx, d.nz, d.dz
    shape = (ny, nx, nz)
    so = _Soil(cfg, shape, dev)
    top = next(b for b in cfg.boundary_conditions if b.target == "groundwater_top")
    head_top = top.kind == "head"
    bath = torch.as_tensor(d.bottom_elevation, dtype=torch.float64, device=dev).expand(ny, nx)
    offset = max(0.0, -float(bath.min()))
    layer = torch.arange(1, nz + 1, device=dev, dtype=torch.float64) * dz
    bot = (bath + offset)[..., None] - layer
    zc = bot + 0.5 * dz
    # Slope metrics of the face toward index + 1 (dx = dy = 1).
    sin, cos, area, up = [], [], [], []
    for axis in (1, 0):
        rise = _shift(zc, axis, 1) - zc
        rise.narrow(axis, shape[axis] - 1, 1).zero_()
        if not d.follow_terrain:
            rise.zero_()
        dist = torch.sqrt(rise * rise + 1.0)
        sin.append(rise.abs() / dist)
        cos.append(1.0 / dist)
        area.append(dz / dist)
        up.append(torch.where(_shift(bot, axis, 1) > bot, 1.0, -1.0))
    vol, ss = dz, g.specific_storage

    def lateral(k, axis):
        """Face conductivity toward index + 1, 0 on the closed edge."""
        f = 0.5 * (k + _shift(k, axis, 1))
        f.narrow(axis, shape[axis] - 1, 1).zero_()
        return f

    def vertical(k, ktop):
        f = torch.empty(ny, nx, nz + 1, dtype=torch.float64, device=dev)
        f[..., 1:nz] = 0.5 * (k[..., 1:] + k[..., :-1])
        f[..., 0] = ktop
        f[..., nz] = k[..., nz - 1]
        return f

    def faces(h):
        kx, kz = so.conductivity(h, so.kx), so.conductivity(h, so.kz)
        return lateral(kx, 1), lateral(kx, 0), vertical(kz, so.kz[..., 0] if head_top else kz[..., 0])

    ic = cfg.initial
    if ic.form == "head":
        h = torch.full(shape, float(ic.value), dtype=torch.float64, device=dev)
    else:
        table = torch.as_tensor(ic.value, dtype=torch.float64, device=dev)
        h = (table + offset)[..., None] - zc
    wc = so.theta(h)
    dt = g.timestep.dt_init
    for _ in range(steps):
        hn, wcn = h, wc
        fx, fy, fz = faces(hn)
        legs = [-f * dt * c * a for f, c, a in zip((fx, fy), cos, area)]
        gz = -fz[..., 1:] * dt / dz
        gz[..., nz - 1] = 0.0  # free drainage: no leg below
        gtop = -2.0 * fz[..., 0] * dt / dz
        storage = so.capacity(hn) + ss * wcn / so.ts
        diag = storage * vol - gz - _shift(gz, 2, -1)
        for leg, axis in zip(legs, (1, 0)):
            diag -= leg + _shift(leg, axis, -1)
        b = storage * hn * vol - dt * fz[..., 1:] + dt * fz[..., :nz]
        for f, a, s, sg, axis in zip((fx, fy), area, sin, up, (1, 0)):
            term = sg * dt * a * f * s
            b += term - _shift(term, axis, -1)
        if head_top:
            diag[..., 0] -= gtop
            b[..., 0] -= gtop * top.value
        else:
            b[..., 0] -= dt * (top.value + fz[..., 0])
        h = _solve(diag, legs[0], legs[1], gz, b, hn)
        fx, fy, fz = faces(h)
        flux = []
        for f, c, a, s, sg, axis in zip((fx, fy), cos, area, sin, up, (1, 0)):
            flux.append(a * (f * c * (_shift(h, axis, 1) - h) + sg * f * s))
        qz = torch.empty_like(fz)
        qz[..., 1:nz] = fz[..., 1:nz] * ((h[..., 1:] - h[..., :-1]) / dz - 1.0)
        qz[..., nz] = -fz[..., nz]
        qz[..., 0] = (so.kz[..., 0] * ((h[..., 0] - top.value) / (0.5 * dz) - 1.0)
                      if head_top else top.value)
        net = qz[..., 1:] - qz[..., :nz]
        for q, axis in zip(flux, (1, 0)):
            net = net + q - _shift(q, axis, -1)
        wc = (wcn * vol + dt * net) / (vol * (1.0 + ss * (h - hn) / so.ts))
        h, wc = _allocate(so, h, wc, fx, fy, fz, vol, dz, qz, dt, head_top and top.value >= 0.0,
                          head_top)
        wc = wc.clamp(so.tr, so.ts)
        qin = flux[0] / area[0] + flux[1] / area[1] + qz[..., 1:]
        qou = _shift(flux[0], 1, -1) / area[0] + _shift(flux[1], 0, -1) / area[1] + qz[..., :nz]
        change = float(((qin - qou).abs() * dt / dz)[..., 1:].max())
        courant = g.timestep.courant_max * dz / so.dk_dtheta(wc)
        limit = float(torch.where(wc < so.ts, courant, torch.full_like(wc, math.inf))[..., 1:].min())
        nxt = dt * (0.75 if change > g.timestep.dq_shrink else
                    1.25 if change < g.timestep.dq_grow else 1.0)
        dt = max(min(nxt, limit, g.timestep.dt_max), g.timestep.dt_min)
    return {"h": h, "wc": wc}


def _solve(diag, gx, gy, gz, b, x):
    """The symmetric 7-point system by Jacobi CG, to rounding."""
    def apply(v):
        out = diag * v
        for leg, axis in ((gx, 1), (gy, 0), (gz, 2)):
            out += leg * _shift(v, axis, 1) + _shift(leg * v, axis, -1)
        return out

    x = x.clone()
    for _ in range(2):  # restarted once: the recurrence's residual drifts
        r = b - apply(x)
        z = r / diag
        p = z.clone()
        rz = (r * z).sum()
        target = 1e-28 * float((b * b / diag).sum())
        for it in range(20000):
            w = apply(p)
            alpha = rz / (p * w).sum()
            x += alpha * p
            r -= alpha * w
            z = r / diag
            new = (r * z).sum()
            if it % 16 == 15 and float(new) <= target:
                break
            p = z + (new / rz) * p
            rz = new
    return x


def _allocate(so, h, wc, fx, fy, fz, vol, dz, qz, dt, wet_top, head_top):
    """The post-allocation on the corrected moisture: saturated cells send
    their excess along the column, cells beside saturation follow theta(h),
    the others h(theta).  qz takes the sends' transfers."""
    nz = h.shape[2]
    sat = (wc >= so.ts) | (h > so.aev)
    beside = torch.zeros_like(sat)
    beside[..., :-1] |= sat[..., 1:]
    beside[..., 1:] |= sat[..., :-1]
    for f, axis in ((fx, 1), (fy, 0)):
        open_ = f != 0.0
        beside |= open_ & _shift(sat, axis, 1)
        beside |= _shift(open_ & sat, axis, -1)
    if wet_top:
        beside[..., 0] = True

    def gradient(axis, f, length, gravity):
        """Head gradients over the faces toward index + 1 and index - 1."""
        plus = torch.where(f > 0.0, (_shift(h, axis, 1) - h) / length - gravity, torch.zeros_like(h))
        minus = torch.where(_shift(f, axis, -1) > 0.0, (h - _shift(h, axis, -1)) / length - gravity,
                            torch.zeros_like(h))
        return plus, minus

    inner = fz[..., 1:].clone()
    inner[..., nz - 1] = 0.0
    total = torch.zeros_like(h)
    for axis, f, length, gravity in ((1, fx, 1.0, 0.0), (0, fy, 1.0, 0.0), (2, inner, dz, 1.0)):
        plus, minus = gradient(axis, f, length, gravity)
        same = plus * minus >= 0.0
        mean = torch.where(same, 0.5 * (plus + minus), torch.zeros_like(h))
        total += torch.where(same, mean.abs(), plus.abs() + minus.abs())
    safe = torch.where(total > 0.0, total, torch.ones_like(total))
    up = torch.where(mean > 0.0, mean, torch.where(mean < 0.0, torch.zeros_like(h), minus.abs()))
    down = torch.where(mean < 0.0, -mean, torch.where(mean > 0.0, torch.zeros_like(h), plus.abs()))
    full = wc >= so.ts
    excess = torch.where(full & (total > 0.0), (wc - so.ts) * vol, torch.zeros_like(wc))
    send_up, send_down = excess * up / safe, excess * down / safe

    dry = ~full & ~beside & (wc < 0.9999 * so.ts)
    follow = ~full & beside
    new_h = torch.where(dry, so.head(wc), h)
    new_wc = torch.where(full, torch.full_like(wc, so.ts), torch.where(follow, so.theta(h), wc))
    room = (so.ts - new_wc) * vol

    def take(left, cell, face, sign):
        got = torch.minimum(room[..., cell].clamp(min=0.0), left)
        new_wc[..., cell] += got / vol
        room[..., cell] -= got
        qz[..., face] += sign * got / dt
        return left - got

    busy_up = (send_up > 0.0).any(0).any(0).tolist()
    busy_down = (send_down > 0.0).any(0).any(0).tolist()
    for k in range(nz):
        if busy_up[k]:
            left = send_up[..., k]
            for cell in range(k - 1, -1, -1):
                left = take(left, cell, cell + 1, 1.0)
            if head_top:
                qz[..., 0] += left / dt
            else:
                for cell in range(1, nz):
                    left = take(left, cell, cell, -1.0)
        if busy_down[k]:
            left = send_down[..., k]
            for cell in range(k + 1, nz):
                left = take(left, cell, cell, -1.0)
    return new_h, new_wc
