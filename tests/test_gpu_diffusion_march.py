"""The 2D explicit diffusion march (31 columns per warp, segments of rows, bc! folded into the
stores) at the edges of its strips and segments."""

import ctypes

import numpy as np
import pytest

from _oracle import NpField, bc_apply, desc_array, lib, vec_fields
from chmy_gb300.bcs import Dirichlet, Neumann, Periodic, to_cg_bc
from chmy_gb300.grids import Center, UniformGrid
from gpu_helpers import assert_close, random_field, to_gpu

pytestmark = pytest.mark.gpu

SPECS = {
    "mixed": {"x": (Dirichlet(0.25), Neumann(-0.3)), "y": (Neumann(0.2), Dirichlet(0.1))},
    "one_sided": {"x": (None, Neumann(0.4)), "y": (Dirichlet(-0.2), None)},
    "periodic_x": {"x": Periodic(), "y": Neumann()},
    "none": None,
}


@pytest.mark.parametrize("T", [np.float32, np.float64])
@pytest.mark.parametrize("dims", [(2, 2), (29, 4), (30, 5), (31, 33), (60, 8), (61, 40)])
@pytest.mark.parametrize("chi", [1.0, 0.7])
@pytest.mark.parametrize("kind", list(SPECS))
@pytest.mark.parametrize("nsteps", [1, 4])
def test_run_equals_oracle(arch, T, dims, chi, kind, nsteps):
    """cg_diffusion_run leaves both buffers with the bits of the oracle's compute_q!, update_C!, bc!(C):
    grids that fill a strip of 31 columns (0..n+1), exceed it by one and end one short; chi = 1 and a
    general chi; rules on both sides, on one side, periodic (not folded) and no bc!."""
    grid = UniformGrid(origin=(T(-1),) * 2, extent=(T(2), T(1.7)), dims=dims, dtype=T)
    C = random_field(grid, Center(), T, np.random.default_rng(3))
    bc = to_cg_bc(2, SPECS[kind]) if kind != "none" else None
    A, B = to_gpu(arch, C), to_gpu(arch, C)
    dt = float(min(grid.spacing())) ** 2 / chi / 8.2
    g, prev = grid.desc(), C.a.copy()
    for _ in range(nsteps):
        prev = C.a.copy()
        q = vec_fields(grid, T)
        lib().or_diffusion_compute_q(ctypes.byref(g), desc_array(q, 3), ctypes.byref(C.desc()), chi)
        lib().or_diffusion_update_C(ctypes.byref(g), ctypes.byref(C.desc()), desc_array(q, 3), dt)
        if bc is not None:
            bc_apply(grid, [C], [bc])
    arch.call("cg_diffusion_run", ctypes.byref(g), ctypes.byref(A.desc()), ctypes.byref(B.desc()), chi, dt,
              ctypes.byref(bc) if bc is not None else None, nsteps)
    last, before = (B, A) if nsteps % 2 else (A, B)
    assert_close(last, C, 0.0, "C^N", exact=True)
    if nsteps > 1:
        ref = NpField(grid, Center(), T)
        ref.a[...] = prev
        assert_close(before, ref, 0.0, "C^(N-1)", exact=True)
