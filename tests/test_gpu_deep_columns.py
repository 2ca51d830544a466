"""The post-allocation of columns around and past the warp walk's depth: wet
hillslopes, whose surplus travels whole columns."""
import numpy as np
import pytest

from frehg_b200 import workloads
from frehg_b200.gw import RichardsSolver
from oracle.gw import OracleSolver

pytestmark = pytest.mark.gpu


# The mixed form's deepest column: a second and more of one thread's walk.  The
# phases timed apart are the same passes, so the states agree bit for bit.
def test_deepest_column():
    cfg = workloads.hillslope(4, 4, 4096, precision="mixed")
    with RichardsSolver(cfg) as s, RichardsSolver(cfg) as apart:
        apart.setProfiling(True)
        for _ in range(2):
            dt = s.nextDt()
            s.step(0.0, dt)
            apart.step(0.0, dt)
        for name in ("h", "wc", "qz"):
            np.testing.assert_array_equal(s.field(name), apart.field(name))


# 352 cells: the last of the warp walk; 353: the first of the thread walk.  In
# lockstep with the oracle at its own rtol, with the parity tests' bar.
@pytest.mark.parametrize("nz", [352, 353])
def test_walk_depths(nz):
    cfg = workloads.hillslope(5, 4, nz)
    with RichardsSolver(cfg) as g:
        o = OracleSolver(cfg)
        try:
            moved = 0.0
            for n in range(3):
                dt = o.next_dt()
                o.step(0.0, dt)
                info = g.step(0.0, dt)
                moved += abs(info["realloc_adjust"])
                for name in ("h", "wc", "qz"):
                    a, b = g.field(name), o.field(name)
                    err = np.max(np.abs(a - b)) / np.max(np.abs(b))
                    assert err <= 1e-9, (n, name, err)
            assert moved > 0.0
        finally:
            o.close()
