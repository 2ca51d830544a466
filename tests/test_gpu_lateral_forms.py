"""The solver forms and field reads on boxes in which every column differs from
its neighbours: conductivities per cell and direction, an initial head that
varies in all three directions, ponding on half of the top.  A value taken from
the wrong column, or through the other direction's leg, shows here.

The bars are those of the uniform boxes: the line forms (outer_rtol 1e-13)
within 1e-9 of the FP64 oracle solved to 1e-13; the FP64 form within 1e-9 of
the oracle at its own rtol, with its iteration count to within two.
"""
import numpy as np
import pytest

from frehg_b200 import workloads
from frehg_b200.config import BoundaryCondition
from frehg_b200.gw import RichardsSolver
from oracle.gw import OracleSolver

pytestmark = pytest.mark.gpu

SMS, THREADS = 148, 512  # a solve's blocks at most, and their threads


def box(nx, ny, nz, precision, rtol):
    rng = np.random.default_rng(nx * 10007 + ny * 101 + nz)
    cfg = workloads.column_32x32x50(nx, ny, nz, precision=precision)
    shape = (ny, nx, nz)
    cell = {name: 1e-5 * np.exp(0.7 * rng.standard_normal(shape)) for name in ("ksx", "ksy", "ksz")}
    cfg.cell_soil = dict(cell, vg_alpha=np.full(shape, 1.0), vg_n=np.full(shape, 2.0))
    cfg.initial.value = -1.0 - 0.5 * rng.random(shape)
    half = [(-0.1, -0.1), (nx + 0.1, -0.1), (nx + 0.1, 0.5 * ny + 0.01), (-0.1, 0.5 * ny + 0.01)]
    cfg.boundary_conditions[0] = BoundaryCondition("pond", half, "groundwater_top", "head",
                                                   "constant", 0.01)
    cfg.solver.rtol, cfg.solver.atol = rtol, 1e-300
    cfg.solver.max_iterations = 20000
    cfg.solver.outer_rtol = 1e-13
    return cfg


def compare(nx, ny, nz, precision, rtol, steps=2, names=("h", "wc")):
    with RichardsSolver(box(nx, ny, nz, precision, rtol)) as g:
        o = OracleSolver(box(nx, ny, nz, "fp64", rtol if precision == "fp64" else 1e-13))
        try:
            for n in range(steps):
                dt = o.next_dt()
                o.step(0.0, dt)
                info = g.step(0.0, dt)
                if precision == "fp64":
                    assert abs(info["cg_iterations"] - o.info["cg_iterations"]) <= 2, n
                for name in names:
                    a, b = g.field(name), o.field(name)
                    err = np.max(np.abs(a - b)) / np.max(np.abs(b))
                    assert err <= 1e-9, (n, name, err)
        finally:
            o.close()


def pairs(nx, ny, nz):
    """Pairs of cells a thread of the FP64 solve takes."""
    cells = (nx + 2) * (ny + 2) * nz
    blocks = min(-(-(cells // 2) // THREADS), SMS)
    return -(-(cells // 2) // (blocks * THREADS))


# One barrier an iteration (1e-10) and two (1e-12) on up to five pairs a thread:
# seven own words in shared memory (1, 2 pairs), four (3, 4), two (5).
@pytest.mark.parametrize("shape,p", [((19, 17, 40), 1), ((19, 17, 41), 1), ((38, 46, 100), 2),
                                     ((38, 46, 101), 2), ((61, 59, 96), 3), ((61, 59, 97), 3),
                                     ((70, 73, 102), 4), ((70, 73, 101), 4), ((80, 83, 102), 5),
                                     ((80, 83, 103), 5)])
@pytest.mark.parametrize("rtol", [1e-10, 1e-12])
def test_fp64_up_to_five_pairs(shape, p, rtol):
    assert pairs(*shape) == p
    compare(*shape, "fp64", rtol)


# Two barriers at every rtol beyond: two own words (6 pairs), one, none.
@pytest.mark.parametrize("shape,p", [((88, 90, 102), 6), ((88, 90, 101), 6), ((120, 118, 112), 11),
                                     ((120, 118, 111), 11), ((150, 149, 114), 18),
                                     ((150, 149, 113), 18)])
def test_fp64_beyond_five_pairs(shape, p):
    assert pairs(*shape) == p
    compare(*shape, "fp64", 1e-10, steps=1)


# Every lanes-per-column form, whole and with one to three cells of padding.
@pytest.mark.parametrize("nz", [1, 2, 3, 5, 31, 32, 33, 63, 66, 127, 128, 130, 201, 255])
@pytest.mark.parametrize("precision", ["mixed", "fp64_line"])
def test_line_depths(nz, precision):
    compare(13, 11, nz, precision, 1e-12)


# Chunked columns (256 cells a chunk); the last two end in a padded chunk and in
# one of a single cell.
@pytest.mark.parametrize("shape", [(9, 7, 257), (9, 7, 385), (5, 6, 767), (3, 2, 4096), (3, 2, 4095),
                                   (2, 3, 3841)])
def test_line_chunks(shape):
    compare(*shape, "mixed", 1e-12, steps=1)


# Columns a warp takes: beside one column's, 3 to 6 (mixed: three own words in
# shared memory, FP64: three up to 3, then none) and 7 (none).
@pytest.mark.parametrize("shape", [(140, 139, 9), (241, 239, 5), (70, 69, 67), (121, 119, 66)])
@pytest.mark.parametrize("precision", ["mixed", "fp64_line"])
def test_line_columns_a_warp(shape, precision):
    compare(*shape, precision, 1e-12, steps=1)


# Fields of 16 KB with their halo, the last to be read whole, and the next.
@pytest.mark.parametrize("nz", [32, 33])
def test_field_kinds(nz):
    compare(6, 6, nz, "fp64", 1e-12, names=("h", "wc", "qx", "qy", "qz", "kx", "ky", "kz"))
