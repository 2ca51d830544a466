"""Parity of the B200 step (through the C ABI) with the CPU oracle.

Bars (stated per test): head within 1e-9 relative L-inf, the other state
and flux fields within 1e-8 of their L-inf scale, CG iteration counts
within +-2 of the oracle's, the GPU's own per-step mass audit closing to
1e-12 of the total storage, and the controller's next dt equal to the
oracle's within 1e-9 relative.
"""
import numpy as np
import pytest

import cases
from frehg_b200 import workloads
from frehg_b200.gw import RichardsSolver
from oracle.gw import OracleSolver

pytestmark = pytest.mark.gpu

H_TOL = 1e-9
F_TOL = 1e-8


# Scale floors of the L-inf comparison: a field whose magnitude is below its
# floor (e.g. rounding-level fluxes of a column at equilibrium) is compared
# absolutely against the floor instead.
FLOOR = {"h": 1.0, "wc": 1.0, "qx": 1e-12, "qy": 1e-12, "qz": 1e-12, "kx": 1e-12,
         "ky": 1e-12, "kz": 1e-12}


FLUX_SCALE = {"qx": ("kx", "ax"), "qy": ("ky", "ay"), "qz": ("kz", None)}


def rel_linf(a, b, floor=0.0):
    if not b.size:
        return 0.0
    scale = max(float(np.max(np.abs(b))), floor)
    if scale == 0.0:
        return float(np.max(np.abs(a)))
    return float(np.max(np.abs(a - b)) / scale)


def compare(cfg, steps, fields=("h", "wc", "qx", "qy", "qz", "kx", "ky", "kz"), t_end=None,
            dt_rtol=1e-9, dt_misses=0.0):
    """Steps the B200 form and the oracle in lockstep on the oracle's dt
    sequence: ``steps`` steps, or, with ``t_end``, the reference driver's
    loop to that time (``Simulation::runGroundwaterLoop``,
    driver/Simulation.cpp:1695-1699: step while t < t_end - 1e-9, the last
    step not clipped).  Returns the CG iteration counts of both.  The GPU's
    own next dt must match the oracle's within dt_rtol on all but a fraction
    dt_misses of the steps."""
    gpu = RichardsSolver(cfg)
    cpu = OracleSolver(cfg)
    try:
        # Geometry is host set-up: bitwise.  The initial state comes from the
        # retention curve, whose pow() differs by ulps between CUDA and glibc.
        for name in ("dz3d", "bot3d", "ax", "ay", "sinx", "cosx", "siny", "cosy"):
            np.testing.assert_array_equal(gpu.field(name), cpu.field(name), err_msg=name)
        for name in ("h", "wc"):
            np.testing.assert_allclose(gpu.field(name), cpu.field(name), rtol=1e-14, atol=1e-15,
                                       err_msg=name)
        prev = gpu.ownedVolume()
        its = []
        misses = 0
        n = 0
        while (n < steps) if t_end is None else (cpu.t < t_end - 1.0e-9):
            dtg = cpu.next_dt()
            if gpu.nextDt() != pytest.approx(dtg, rel=dt_rtol):
                misses += 1
                assert misses <= dt_misses * max(n, 1), f"next dt step {n}: {gpu.nextDt()} vs {dtg}"
            cpu.t += dtg
            cpu.step(cpu.t, dtg)
            info = gpu.step(cpu.t, dtg)
            its.append((info["cg_iterations"], cpu.info["cg_iterations"]))
            assert abs(info["cg_iterations"] - cpu.info["cg_iterations"]) <= 2, f"step {n}"
            assert rel_linf(gpu.field("h"), cpu.field("h"), FLOOR["h"]) <= H_TOL, f"h step {n}"
            for name in fields[1:]:
                ref = cpu.field(name)
                floor = FLOOR[name]
                if name in FLUX_SCALE:
                    # A net Darcy flux is a difference of a pressure and a
                    # gravity term; near equilibrium it cancels to the solve's
                    # residual, so its error is measured on the gravity scale
                    # K * A of that direction.
                    kname, area = FLUX_SCALE[name]
                    a = cfg.domain.dx * cfg.domain.dy if area is None else cpu.field(area)
                    floor = max(floor, float(np.max(np.abs(cpu.field(kname)) * a)))
                err = rel_linf(gpu.field(name), ref, floor)
                assert err <= F_TOL, f"{name} step {n}: {err}"
            v = gpu.ownedVolume()
            resid = (v - prev) - (info["boundary_in"] - info["ss_storage"] +
                                  info["realloc_adjust"] - info["vloss"])
            assert abs(resid) <= 1e-12 * max(v, 1.0), f"audit step {n}: {resid}"
            assert v == pytest.approx(cpu.owned_volume(), rel=1e-10)
            prev = v
            n += 1
        assert misses <= dt_misses * n
    finally:
        gpu.close()
    return its


@pytest.mark.parametrize("name", sorted(cases.SCENARIOS))
def test_scenario_parity(name):
    compare(cases.SCENARIOS[name](), 8)


def test_box_32x32x50_parity():
    compare(workloads.column_32x32x50(), 6)


def test_hillslope_crop_parity():
    compare(workloads.hillslope(24, 20, 32), 4)


def test_box_32x32x50_to_end_time():
    # The homogeneous box case as described: 1 h of simulated time from
    # dt0 = 10 s (about 300 adaptive steps, 8 to 40 CG iterations each).  Once
    # the wetting front nears saturation the controller's Courant cap
    # Co dz / (dK/dtheta) over the unsaturated cells sets dt.  dK/dtheta there
    # amplifies the last bits of theta by 1 / (1 - Se^(1/m)), and whether a
    # cell the post-allocation leaves at theta_s counts as unsaturated is
    # decided by its last bit, so the cap is discontinuous: the GPU's own next
    # dt (from its own state; the steps take the oracle's dt) is held to 1e-8
    # on all but 5 % of the steps, and every step meets the head, field, CG
    # and audit bars.
    its = compare(workloads.column_32x32x50(), 0, t_end=3600.0, dt_rtol=1e-8, dt_misses=0.05)
    assert len(its) > 100


def test_slab_crop_64x64x128_parity():
    # The benchmark slab's construction at its column depth and spacing
    # (nz = 128, dz = 0.05 m, terrain-following, per-cell soil) on a
    # 64x64 footprint, 10 steps: the first 60 s step takes ~1600 Jacobi-CG
    # iterations and the later ones ~360, so the +-2 iteration and 1e-9 head
    # bars hold where FMA rounding has the most iterations to drift.
    its = compare(workloads.hillslope(64, 64, 128), 10)
    assert max(o for _, o in its) > 1000


def test_deep_columns_parity():
    # Warp walks of 190 cells, which need more than the default 48 KB of shared
    # memory per block, and of 257.
    compare(workloads.column_32x32x50(nx=3, ny=2, nz=190), 3)
    compare(workloads.column_32x32x50(nx=2, ny=2, nz=257), 2)


def test_step_is_deterministic():
    cfg = cases.mixed_box()
    runs = []
    for _ in range(2):
        with RichardsSolver(cfg) as g:
            for _ in range(5):
                g.advance()
            runs.append((g.field("h"), g.field("wc"), g.field("qz"), g.nextDt()))
    for a, b in zip(runs[0], runs[1]):
        np.testing.assert_array_equal(a, b)


def test_invalid_step_is_rejected():
    from frehg_b200.gw import FatalError
    with RichardsSolver(cases.closed_column()) as g:
        with pytest.raises(FatalError):
            g.step(1.0, -1.0)


def test_cg_iteration_cap_reports_divergence():
    # max_iterations = 1 cannot reach rtol on the 32x32x50 box: the reference
    # treats KSP_DIVERGED_ITS as fatal; the ABI returns FREHG_GW_ESOLVER.
    from frehg_b200.gw import FatalError
    cfg = workloads.column_32x32x50(nx=8, ny=8, nz=20)
    cfg.solver.max_iterations = 1
    with RichardsSolver(cfg) as g:
        with pytest.raises(FatalError) as e:
            g.advance()
        assert e.value.status == 5


def test_partial_boundary_updates_match_oracle():
    # updateBoundaryValues with some slots only (None keeps the others): the
    # upload sends the top and bottom slots and the sides' edge entries, and
    # the step must follow the oracle given the same updates.
    cfg = cases.SCENARIOS["side_flux"]()
    d = cfg.domain
    gpu = RichardsSolver(cfg)
    cpu = OracleSolver(cfg)
    rng = np.random.default_rng(9)
    try:
        updates = [dict(top=-1e-6 * (1.0 + rng.random((d.ny, d.nx)))),
                   dict(xm=2e-6 * rng.random(d.ny), xp=-1e-6 * rng.random(d.ny)),
                   dict(ym=1e-6 * rng.random(d.nx)),
                   dict(yp=-2e-6 * rng.random(d.nx), bottom=np.zeros((d.ny, d.nx))),
                   dict()]
        for n, u in enumerate(updates):
            gpu.setBoundaryValues(**u)
            cpu.set_boundary_values(**u)
            dtg = cpu.next_dt()
            cpu.t += dtg
            cpu.step(cpu.t, dtg)
            gpu.step(cpu.t, dtg)
            assert rel_linf(gpu.field("h"), cpu.field("h"), 1.0) <= H_TOL, f"h step {n}"
            for name in ("qx", "qy", "qz"):
                kname, area = FLUX_SCALE[name]
                a = d.dx * d.dy if area is None else cpu.field(area)
                floor = max(1e-12, float(np.max(np.abs(cpu.field(kname)) * a)))
                assert rel_linf(gpu.field(name), cpu.field(name), floor) <= F_TOL, f"{name} {n}"
    finally:
        gpu.close()


def test_handle_records_its_device():
    import ctypes

    import torch
    with RichardsSolver(cases.closed_column()) as g:
        g.lib.frehg_gw_device.restype = ctypes.c_int
        g.lib.frehg_gw_device.argtypes = [ctypes.c_void_p]
        assert g.lib.frehg_gw_device(g.h) == torch.cuda.current_device()


def test_rejected_boundary_update_changes_nothing():
    # A non-finite value is refused with EINVAL and leaves the domain as it
    # was: the steps after it equal those of a twin that never saw it.
    from frehg_b200.gw import FatalError
    cfg = cases.SCENARIOS["side_flux"]()
    d = cfg.domain
    a, b = RichardsSolver(cfg), RichardsSolver(cfg)
    try:
        bad_top = np.full((d.ny, d.nx), -1e-6)
        bad_top[-1, -1] = np.nan
        bad_xm = np.full(d.ny, 1e-6)
        bad_xm[0] = np.inf
        with pytest.raises(FatalError) as e:
            a.setBoundaryValues(top=bad_top, xm=bad_xm)
        assert e.value.status == 1
        good = dict(ym=1e-6 * np.ones(d.nx))
        a.setBoundaryValues(**good)
        b.setBoundaryValues(**good)
        for _ in range(3):
            a.advance()
            b.advance()
        np.testing.assert_array_equal(a.field("h"), b.field("h"))
        np.testing.assert_array_equal(a.field("qx"), b.field("qx"))
    finally:
        a.close()
        b.close()
