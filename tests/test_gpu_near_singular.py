"""The one-barrier form of the FP64 solve on systems close to singular: closed
saturated boxes whose specific storage is next to nothing keep their volume, so
their mean head, whatever the flow inside does.  What a solve does to the mean
is the distance of its last residual from the one it believes in, times the
condition number (1e9 and more here).

The bar is ten times what the two-barrier form of the same system does (at
rtol 9e-11, the other side of the dispatch): the two round differently, and both
are CG with the residual taken from A p."""
import numpy as np
import pytest

from frehg_b200.config import (Domain, Groundwater, GwConfig, InitialCondition, Solver, SoilType,
                               Timestep)
from frehg_b200.gw import RichardsSolver

pytestmark = pytest.mark.gpu


def drift(nx, ny, nz, rtol):
    rng = np.random.default_rng(5)
    shape = (ny, nx, nz)
    head = 1.0 + rng.random(shape)
    ks = 1e-5 * np.exp(rng.standard_normal(shape))
    cfg = GwConfig(
        domain=Domain(nx=nx, ny=ny, nz=nz, dx=10.0, dy=10.0, dz=0.02, bottom_elevation=0.0),
        soil_types=[SoilType("s", 1e-5, 1e-5, 1e-5, 0.4, 0.05, 1.0, 2.0, 0.0)],
        groundwater=Groundwater(timestep=Timestep(dt_init=600.0, dt_min=600.0, dt_max=600.0),
                                specific_storage=1e-9),
        initial=InitialCondition("head", head),
        solver=Solver(rtol=rtol, atol=1e-300, max_iterations=50000),
        cell_soil=dict(ksx=ks, ksy=ks, ksz=ks))
    with RichardsSolver(cfg) as s:
        s.step(0.0, 600.0)
        return abs(s.head().mean() - head.mean())


@pytest.mark.parametrize("shape", [(20, 20, 20), (21, 19, 23), (40, 40, 40)])
def test_volume_of_a_closed_box(shape):
    assert drift(*shape, 1e-10) <= 10.0 * max(drift(*shape, 9e-11), 1e-8)
