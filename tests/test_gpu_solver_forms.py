"""The forms of the predictor solves at the sizes where their dispatch and
their layouts can go wrong: column depths around the lanes-per-column and
chunk limits of the line solves, odd cell counts and single blocks of the FP64
solve, the sizes on either side of its shared-memory and one-barrier rules,
and steps on either side of the small-domain launches.

Each domain takes three steps of the box.  The line forms (outer_rtol 1e-13)
follow the FP64 oracle solved tightly (rtol 1e-13): a residual of 1e-13 times
the box's conditioning, below 1e3 at these steps, stays under 1e-9 relative
with an order to spare.  The FP64 form has the oracle's algorithm, so it
follows the oracle at its own rtol, in lockstep, with the parity tests' bars:
1e-9 relative and the oracle's iteration count to within two.  Fields read
back through the packed read are compared with what was set, exactly.
"""
import threading

import numpy as np
import pytest

from frehg_b200 import workloads
from frehg_b200.gw import RichardsSolver
from oracle.gw import OracleSolver

pytestmark = pytest.mark.gpu

STEPS = 3


def box(nx, ny, nz, precision, rtol):
    cfg = workloads.column_32x32x50(nx, ny, nz, precision=precision)
    cfg.solver.rtol = rtol
    cfg.solver.atol = 1e-300
    cfg.solver.max_iterations = 20000
    cfg.solver.outer_rtol = 1e-13
    return cfg


def compare(nx, ny, nz, precision, rtol):
    g = RichardsSolver(box(nx, ny, nz, precision, rtol))
    o = OracleSolver(box(nx, ny, nz, "fp64", rtol if precision == "fp64" else 1e-13))
    try:
        for n in range(STEPS):
            dt = o.next_dt()
            o.step(0.0, dt)
            info = g.step(0.0, dt)
            if precision == "fp64":
                assert abs(info["cg_iterations"] - o.info["cg_iterations"]) <= 2, n
            for name in ("h", "wc"):
                a, b = g.field(name), o.field(name)
                err = np.max(np.abs(a - b)) / np.max(np.abs(b))
                assert err <= 1e-9, (n, name, err)
    finally:
        g.close()
        o.close()


# 1, 33, 65, 129: the first depth of each column variant (257 below); 32, 64,
# 128, 256: the last; others leave a padded quad.
@pytest.mark.parametrize("nz", [1, 3, 32, 33, 64, 65, 127, 128, 129, 256])
@pytest.mark.parametrize("precision", ["mixed", "fp64_line"])
def test_column_depths(nz, precision):
    compare(5, 3, nz, precision, 1e-12)


@pytest.mark.parametrize("nz", [257, 511, 512, 513, 1025])
def test_deep_columns(nz):
    compare(3, 2, nz, "mixed", 1e-12)


# One column, one block, a block's last warp alone, more than one column a warp.
@pytest.mark.parametrize("nx,ny", [(1, 1), (16, 1), (17, 1), (1, 33), (40, 41)])
@pytest.mark.parametrize("precision", ["mixed", "fp64_line"])
def test_column_counts(nx, ny, precision):
    compare(nx, ny, 20, precision, 1e-12)


# Odd and even cell counts; one block, and one to three pairs a thread on more
# (seven or four words in shared memory); one barrier (1e-10) and two (1e-12).
@pytest.mark.parametrize("shape", [(1, 1, 1), (1, 1, 5), (4, 3, 7), (13, 11, 9), (31, 29, 51),
                                   (64, 48, 63), (80, 50, 100)])
@pytest.mark.parametrize("rtol", [1e-10, 1e-12])
def test_fp64_forms(shape, rtol):
    compare(*shape, "fp64", rtol)


# Either side of the small-domain launches (600,000 cells with ghosts).
@pytest.mark.parametrize("nx", [72, 75])
def test_small_domain_boundary(nx):
    compare(nx, 78, 100, "mixed", 1e-12)


# The packed read: below and above the threaded copies, odd sizes, a z-face
# field larger than the cells, two readers at once.
@pytest.mark.parametrize("shape", [(1, 1, 1), (300, 3, 1), (5, 4, 7), (101, 103, 105)])
def test_field_reads(shape):
    nx, ny, nz = shape
    rng = np.random.default_rng(1)
    s = RichardsSolver(workloads.column_32x32x50(nx, ny, nz))
    t = RichardsSolver(workloads.column_32x32x50(nx, ny, nz))
    try:
        want = {}
        for x in (s, t):
            h, wc = -rng.random((ny, nx, nz)), 0.1 + 0.2 * rng.random((ny, nx, nz))
            x.setState(h, wc)
            want[x] = (h, wc)
        got = {}

        def read(x):
            got[x] = (x.head(), x.waterContent())

        threads = [threading.Thread(target=read, args=(x,)) for x in (s, t)]
        [th.start() for th in threads]
        [th.join() for th in threads]
        for x in (s, t):
            for a, b in zip(got[x], want[x]):
                np.testing.assert_array_equal(a, b)
        assert s.field("qz").shape == (ny, nx, nz + 1)
        assert np.all(s.field("qz") == 0.0)
    finally:
        s.close()
        t.close()
