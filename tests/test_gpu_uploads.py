"""What a caller hands over from pageable memory is what the next kernel sees,
also while other transfers keep the copy engine busy: an upload is ordered
before the kernels that read it, not merely issued before them.
"""
import ctypes as C

import numpy as np
import pytest

import cases
from frehg_b200 import workloads
from frehg_b200.config import IC_FORMS
from frehg_b200.gw import RichardsSolver

pytestmark = pytest.mark.gpu

_dp = C.POINTER(C.c_double)


class CopyTraffic:
    """Host-to-device copies on a stream of their own: 1 GiB, some 20 ms."""

    def __init__(self):
        import torch

        self.torch = torch
        self.stream = torch.cuda.Stream()
        self.host = torch.empty(256 << 20, dtype=torch.uint8).pin_memory()
        self.dev = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")

    def start(self):
        with self.torch.cuda.stream(self.stream):
            for _ in range(4):
                self.dev.copy_(self.host, non_blocking=True)

    def wait(self):
        self.torch.cuda.synchronize()


@pytest.fixture(scope="module")
def traffic():
    return CopyTraffic()


# Below, within and above the driver's staging chunks.
@pytest.mark.parametrize("shape", [(8, 6, 20), (32, 32, 50), (23, 10, 353), (100, 100, 100)])
def test_initial_field(shape, traffic):
    nx, ny, nz = shape
    rng = np.random.default_rng(0)
    with RichardsSolver(workloads.column_32x32x50(nx, ny, nz)) as s:
        for n in range(4):
            head = -1.0 - rng.random((ny, nx, nz))
            traffic.start()
            rc = s.lib.frehg_gw_init_state(s.h, IC_FORMS["head"], 0.0, head.ctypes.data_as(_dp))
            traffic.wait()
            assert rc == 0
            np.testing.assert_array_equal(s.head(), head, err_msg=str(n))


def test_scalars(traffic):
    nx, ny, nz = 20, 18, 40
    cfg = cases.mixed_box(nx=nx, ny=ny, nz=nz)
    names = ("salt", "salt_surf")
    with RichardsSolver(cfg) as busy, RichardsSolver(cfg) as idle:
        for s in (busy, idle):
            s.attachDensity(saline=True)
        for n in range(4):
            values = dict(zip(names, cases.density_scalars(nx, ny, nz, step=n)))
            for s in (busy, idle):
                # The cell field last: the step comes right behind its upload.
                s.setScalar("salt_surf", values["salt_surf"])
                if s is busy:
                    traffic.start()
                s.setScalar("salt", values["salt"])
                if s is idle:
                    traffic.wait()
                s.step(0.0, 1.0)
                traffic.wait()
            np.testing.assert_array_equal(busy.field("rho"), idle.field("rho"), err_msg=str(n))
            np.testing.assert_array_equal(busy.head(), idle.head(), err_msg=str(n))


@pytest.mark.parametrize("precision", ["mixed", "fp64_line"])
def test_restored_start(precision, traffic):
    """A checkpoint restored under copy traffic continues bit for bit (the
    previous start head is the last upload before the step)."""
    cfg = workloads.column_32x32x50(30, 31, 40, precision=precision)
    with RichardsSolver(cfg) as s, RichardsSolver(cfg) as t:
        for _ in range(3):
            s.advance()
        ck = s.checkpoint()
        assert "h_prev" in ck
        s.advance()
        for _ in range(3):
            traffic.start()
            t.restore(ck)
            t.advance()
            traffic.wait()
            for name in ("h", "wc", "vloss"):
                np.testing.assert_array_equal(t.field(name), s.field(name))
