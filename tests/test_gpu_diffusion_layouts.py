"""Every layout that the 2D explicit diffusion march is timed over, fixed by CG_DIFFUSION_LAYOUT."""

import ctypes

import numpy as np
import pytest

from _oracle import bc_apply, desc_array, lib, vec_fields
from chmy_gb300.bcs import to_cg_bc
from chmy_gb300.grids import Center, UniformGrid
from gpu_helpers import assert_close, random_field, to_gpu
from test_gpu_diffusion_march import SPECS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [np.float32, np.float64])
@pytest.mark.parametrize("dims", [(30, 5), (61, 40), (93, 51)])
@pytest.mark.parametrize("kind", ["mixed", "one_sided", "none"])
@pytest.mark.parametrize("chi", [1.0, 0.7])
def test_layouts_equal_oracle(arch, monkeypatch, T, dims, kind, chi):
    """Four steps of cg_diffusion_run, and one of cg_diffusion_step, leave the oracle's bits with every
    segment length and both kinds of launch: segments longer than the grid, with a remainder of one row, and
    with the upper boundary inside (dims[1] + 2 rows without rules)."""
    grid = UniformGrid(origin=(T(-1),) * 2, extent=(T(2), T(1.7)), dims=dims, dtype=T)
    C0 = random_field(grid, Center(), T, np.random.default_rng(3))
    bc = to_cg_bc(2, SPECS[kind]) if kind != "none" else None
    pbc = ctypes.byref(bc) if bc is not None else None
    dt = float(min(grid.spacing())) ** 2 / chi / 8.2
    g = grid.desc()
    ref = random_field(grid, Center(), T, np.random.default_rng(3))
    states = []
    for _ in range(4):
        q = vec_fields(grid, T)
        lib().or_diffusion_compute_q(ctypes.byref(g), desc_array(q, 3), ctypes.byref(ref.desc()), chi)
        lib().or_diffusion_update_C(ctypes.byref(g), ctypes.byref(ref.desc()), desc_array(q, 3), dt)
        if bc is not None:
            bc_apply(grid, [ref], [bc])
        states.append(ref.a.copy())
    for seg in (1, 2, 3, 4, 6, 8, 12, 16, 24):
        for dep in (0, 1):
            monkeypatch.setenv("CG_DIFFUSION_LAYOUT", f"{seg}:{dep}")
            A, B = to_gpu(arch, C0), to_gpu(arch, C0)
            arch.call("cg_diffusion_run", ctypes.byref(g), ctypes.byref(A.desc()), ctypes.byref(B.desc()), chi, dt, pbc, 4)
            ref.a[...] = states[3]
            assert_close(A, ref, 0.0, f"{seg}:{dep}", exact=True)
            ref.a[...] = states[2]
            assert_close(B, ref, 0.0, f"{seg}:{dep}, one step earlier", exact=True)
            A, B = to_gpu(arch, C0), to_gpu(arch, C0)
            arch.call("cg_diffusion_step", ctypes.byref(g), ctypes.byref(B.desc()), ctypes.byref(A.desc()), chi, dt, pbc)
            ref.a[...] = states[0]
            assert_close(B, ref, 0.0, f"{seg}:{dep}, one step", exact=True)
