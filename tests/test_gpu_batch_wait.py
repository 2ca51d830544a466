"""A member of a batched solve may wait for the blocks of another member as
long as that one's solve takes.

Two saturated chains of cells in one row (no boundary, condition number 1e7:
some 3,600 iterations a decade of the residual) are stepped at rtol 0 under an
iteration cap, so each solve is exactly that many iterations, some 3 s.
Their blocks are more than half of the device's each: the second chain's first
blocks wait for the first chain to end.  Both have to end at the cap."""
import numpy as np
import pytest

from frehg_b200.abi import StepInfo
from frehg_b200.batch import RichardsBatch
from frehg_b200.config import (Domain, Groundwater, GwConfig, InitialCondition, Solver, SoilType,
                               Timestep)
from frehg_b200.gw import RichardsSolver

pytestmark = pytest.mark.gpu

CELLS, BLOCKS, ITERATIONS = 60000, 100, 300000


def chain(seed):
    rng = np.random.default_rng(seed)
    return GwConfig(
        domain=Domain(nx=CELLS, ny=1, nz=1, dx=1.0, dy=1.0, dz=1.0, bottom_elevation=0.0),
        soil_types=[SoilType("s", 1e-5, 1e-5, 1e-5, 0.4, 0.05, 1.0, 2.0, 0.0)],
        groundwater=Groundwater(timestep=Timestep(dt_init=600.0, dt_min=600.0, dt_max=600.0),
                                specific_storage=2.4e-9),
        initial=InitialCondition("head", 1.0 + rng.random((1, CELLS, 1))),
        solver=Solver(rtol=0.0, atol=0.0, max_iterations=ITERATIONS))


def test_wait_for_another_members_solve():
    members = [RichardsSolver(chain(n)) for n in range(2)]
    with RichardsBatch(members, cells_per_block=CELLS // BLOCKS) as b:
        assert b.solve_blocks() == [BLOCKS, BLOCKS]
        infos = (StepInfo * 2)()
        b.lib.frehg_gw_batch_step(b.b, infos)
        out = [i.as_dict() for i in infos]
    for m in members:
        m.close()
    assert [i["cg_iterations"] for i in out] == [ITERATIONS] * 2
    assert [i["status"] for i in out] == [5, 5]  # the cap, not a barrier that gave up (4)
