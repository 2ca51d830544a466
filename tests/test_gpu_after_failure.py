"""A solver whose step failed on bad data steps on as a new one does once it
has good data again: nothing of the failed solve stays behind."""
import numpy as np
import pytest

import cases
from frehg_b200 import workloads
from frehg_b200.batch import RichardsBatch
from frehg_b200.gw import FatalError, RichardsSolver

pytestmark = pytest.mark.gpu

FIELDS = ("h", "wc", "qx", "qy", "qz")


def closed_cell(precision):
    cfg = workloads.column_32x32x50(1, 1, 1, precision=precision)
    cfg.boundary_conditions = []
    return cfg


def masked_box(precision):
    cfg = cases.mixed_box(nx=9, ny=7, nz=13)
    cfg.solver.precision = precision
    return cfg


def deep_box(precision):
    """Past one block, odd depth; FP64 at 1e-12: two barriers an iteration."""
    cfg = cases.mixed_box(nx=31, ny=29, nz=51)
    cfg.solver.precision = precision
    cfg.solver.rtol = 1e-12
    return cfg


def wide_box(precision):
    """Past one block; FP64 at 1e-8: one barrier an iteration."""
    cfg = cases.mixed_box(nx=31, ny=29, nz=51)
    cfg.solver.precision = precision
    return cfg


BOXES = [closed_cell, masked_box, deep_box, wide_box]


def bad_heads(head):
    """A NaN in one cell; heads whose squares overflow FP32 and FP64."""
    nan = head.copy()
    nan[0, 0, 0] = np.nan
    huge = np.where(np.arange(head.size).reshape(head.shape) % 2, 1e39, -1e39)
    return {"nan": nan, "float": huge, "double": 1e200 * huge / 1e39}


@pytest.mark.parametrize("box", BOXES)
@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp64_line"])
def test_step_after_failed_step(box, precision):
    with RichardsSolver(box(precision)) as s, RichardsSolver(box(precision)) as new:
        head, wc = s.head(), s.waterContent()
        new.setState(head, wc)
        new.step(0.0, 1.0)
        want = {name: new.field(name) for name in FIELDS}
        for what, bad in bad_heads(head).items():
            s.setState(bad, wc)
            try:
                s.step(0.0, 1.0)
            except FatalError:
                pass
            s.setState(head, wc)
            s.step(0.0, 1.0)
            for name in FIELDS:
                np.testing.assert_array_equal(s.field(name), want[name], err_msg=f"{what} {name}")


# A lateral conductivity below zero makes the matrix indefinite under a positive
# diagonal.  The iterations at which the curvature changes sign, even and odd.
@pytest.mark.parametrize("ks,iterations", [(-1.2e-4, 8), (-1.3e-4, 7), (-1.4e-4, 6), (-1.5e-4, 5),
                                           (-1.8e-4, 4), (-2.0e-4, 3)])
def test_iterate_of_an_indefinite_solve(ks, iterations):
    """The two forms of the FP64 solve end at the same iterate: the fluxes, which
    are taken from it, agree to the parity bar."""
    flux = {}
    for rtol in (1e-10, 1e-11):  # one barrier an iteration, two
        cfg = workloads.column_32x32x50(24, 20, 18)
        cfg.soil_types[0].ksx = cfg.soil_types[0].ksy = ks
        cfg.solver.rtol, cfg.solver.atol = rtol, 1e-300
        cfg.initial.value = -1.0 - np.random.default_rng(3).random((20, 24, 18))
        with RichardsSolver(cfg) as s:
            with pytest.raises(FatalError) as e:
                s.step(0.0, 100.0)
            assert f"after {iterations} iterations (KSP reason -10)" in str(e.value)
            flux[rtol] = [s.field(name) for name in ("qx", "qy", "qz")]
    for a, b in zip(flux[1e-10], flux[1e-11]):
        assert np.max(np.abs(a - b)) <= 1e-9 * np.max(np.abs(a))


@pytest.mark.parametrize("precision", ["mixed", "fp64_line"])
def test_exact_start_after_overflow(precision):
    """At rest (head 0 everywhere, no boundary) the first residual is exactly 0
    and the inner solve ends before it has a direction: no earlier step's may be
    added.  Heads over the whole range in which some FP32 value of an iteration
    overflows (factors of 1.5 apart; a product exceeds its factors by 2)."""
    cfg = workloads.column_32x32x50(6, 5, 1, precision=precision)
    cfg.boundary_conditions = []
    rest = np.zeros((5, 6, 1))
    full = np.full((5, 6, 1), 0.40)
    sign = np.where(np.arange(30).reshape(5, 6, 1) % 2, 1.0, -1.0)
    with RichardsSolver(cfg) as s:
        for scale in 1e30 * 1.5 ** np.arange(100):
            s.setState(scale * sign, full)
            try:
                s.step(0.0, 600.0)
            except FatalError:
                pass
            s.setState(rest, full)
            s.step(0.0, 600.0)
            np.testing.assert_array_equal(s.head(), rest, err_msg=str(scale))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_batch_after_failed_step(precision):
    def step(solvers, batch, heads, wcs):
        for s, h, w in zip(solvers, heads, wcs):
            s.setState(h, w)
        for i in range(len(solvers)):
            batch.set_dt(i, 1.0)
        batch.step()

    solvers = [RichardsSolver(box(precision)) for box in BOXES]
    fresh = [RichardsSolver(box(precision)) for box in BOXES]
    heads, wcs = [s.head() for s in solvers], [s.waterContent() for s in solvers]
    with RichardsBatch(solvers) as b, RichardsBatch(fresh) as f:
        step(fresh, f, heads, wcs)
        for what in ("nan", "float", "double"):
            try:
                step(solvers, b, [bad_heads(h)[what] for h in heads], wcs)
            except FatalError:
                pass
            step(solvers, b, heads, wcs)
            for m, (s, n) in enumerate(zip(solvers, fresh)):
                for name in FIELDS:
                    np.testing.assert_array_equal(s.field(name), n.field(name),
                                                  err_msg=f"{what} {m} {name}")
    for s in solvers + fresh:
        s.close()
