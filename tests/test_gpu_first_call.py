"""What the first call at a shape costs: the autotuners' launches, which a program that runs many sizes
once pays every time."""

import ctypes
import time

import numpy as np
import pytest

from chmy_gb300 import Field
from chmy_gb300.bcs import Neumann, to_cg_bc
from chmy_gb300.grids import Center, UniformGrid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,limit_ms", [(120, 3.0), (1000, 8.0)])
def test_first_diffusion_run_at_a_size(arch, n, limit_ms):
    """50 explicit steps at sizes that no call has seen (the median of five, after one that loads the
    kernels): about 1 ms at 120^2 and 3 ms at 1000^2 on GB300. Timing every candidate over 28 launches took
    4.7 and 16.9 ms."""
    import torch

    took = []
    for k in range(6):
        dims = (n + 1 + 2 * k, n + 2 + 2 * k)
        grid = UniformGrid(origin=(-1.0, -1.0), extent=(2.0, 2.0), dims=dims, dtype=np.float64)
        A, B = (Field(arch, grid, Center()) for _ in range(2))
        g, a, b, bc = grid.desc(), A.desc(), B.desc(), to_cg_bc(2, Neumann())
        dt = float(min(grid.spacing())) ** 2 / 8.2
        torch.cuda.synchronize()
        t = time.perf_counter()
        arch.call("cg_diffusion_run", ctypes.byref(g), ctypes.byref(a), ctypes.byref(b), 1.0, dt, ctypes.byref(bc), 50)
        arch.synchronize()
        took.append(1e3 * (time.perf_counter() - t))
    assert sorted(took[1:])[2] < limit_ms, took
