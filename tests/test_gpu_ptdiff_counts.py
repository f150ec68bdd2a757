"""3D FP32 runs of few iterations in the dense layout: copying C and q to partner buffers and back costs
more than the fused iteration saves, and the run takes the flux and update kernels in place."""

import ctypes

import numpy as np
import pytest

from chmy_gb300 import Field, _abi
from chmy_gb300.bcs import Dirichlet, Neumann, to_cg_bc
from chmy_gb300.configs import ptdiff_params
from chmy_gb300.grids import Center, UniformGrid, Vertex

pytestmark = pytest.mark.gpu
T = np.float32


@pytest.mark.parametrize("nsteps,npt,in_place", [(1, 1, True), (3, 1, True), (1, 2, True), (1, 3, True), (1, 4, False), (3, 2, False)])
def test_few_iterations_run_in_place(arch, nsteps, npt, in_place):
    """In place a run has the bits of its launches one by one; the fused iteration rounds every operation by
    itself and differs from them in the last places."""
    dims = (45, 34, 27)
    grid = UniformGrid(origin=(T(-0.5),) * 3, extent=(T(1),) * 3, dims=dims, dtype=T)
    g, bc = grid.desc(), to_cg_bc(3, {"x": Dirichlet(0.1), "y": Neumann(), "z": Neumann(0.2)})
    p = ptdiff_params(grid, 1e-3, 1.5)

    def make():
        rng = np.random.default_rng(11)
        C, C_old, D = (Field(arch, grid, Center(), T) for _ in range(3))
        q = [Field(arch, grid, tuple(Vertex() if e == d else Center() for e in range(3)), T) for d in range(3)]
        for f in [C, D] + q:
            f.from_numpy(rng.uniform(0.5, 1.5, tuple(reversed(f.ext))).astype(T))
        C_old.data.copy_(C.data)
        s = _abi.cg_ptdiff_fields()
        s.C, s.C_old, s.D = C.desc(), C_old.desc(), D.desc()
        s.q = (_abi.cg_field * 3)(*[f.desc() for f in q])
        return s, [C, C_old] + q

    run, a = make()
    arch.call("cg_ptdiff_run", ctypes.byref(g), ctypes.byref(run), ctypes.byref(p), ctypes.byref(bc), nsteps, npt)
    apart, b = make()
    for _ in range(nsteps):
        b[1].data.copy_(b[0].data)
        for _ in range(npt):
            arch.call("cg_ptdiff_update_q", ctypes.byref(g), ctypes.byref(apart), ctypes.byref(p))
            arch.call("cg_ptdiff_update_C", ctypes.byref(g), ctypes.byref(apart), ctypes.byref(p))
            arch.call("cg_bc_apply", ctypes.byref(g), 1, ctypes.byref(apart.C), ctypes.byref(bc))
        arch.synchronize()
    same = all(np.array_equal(x.to_numpy(), y.to_numpy()) for x, y in zip(a, b))
    assert same == in_place
    for x, y in zip(a, b):
        assert np.max(np.abs(x.to_numpy() - y.to_numpy())) <= 2e-5 * nsteps * npt * np.max(np.abs(y.to_numpy()))
