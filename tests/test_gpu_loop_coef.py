"""FP64 loops that compute their coefficients once (viscosity terms of the Stokes loops, face diffusivities
of PT diffusion): when they do, and how far their results are from those of the launches one by one."""

import ctypes

import numpy as np
import pytest

import test_gpu_block_shapes as shapes
from chmy_gb300 import Field, _abi
from chmy_gb300.bcs import Dirichlet, Neumann, to_cg_bc
from chmy_gb300.configs import ptdiff_params
from chmy_gb300.grids import Center, UniformGrid, Vertex
from gpu_helpers import rtol_for
from test_gpu_stokes import StokesSet, _bc_V, pt_params

pytestmark = pytest.mark.gpu
T = np.float64


def stokes(arch, dims, calls):
    """V, P and tau after the calls' iterations (0: one iteration by its launches)."""
    s = StokesSet(arch, dims, T, 43, True)
    p, barr = pt_params(s.grid, True), (_abi.cg_bc * 3)(*_bc_V(len(dims)))
    g, d = s.grid.desc(), s.dev_desc()
    vel = (_abi.cg_field * 3)(*[f.desc() for f in s.d["V"]])
    for n in calls:
        if n:
            arch.call("cg_stokes_pt_iterations", ctypes.byref(g), ctypes.byref(d), ctypes.byref(p), barr, n)
            continue
        arch.call("cg_stokes_update_stress", ctypes.byref(g), ctypes.byref(d), ctypes.byref(p))
        arch.call("cg_stokes_update_velocity", ctypes.byref(g), ctypes.byref(d), ctypes.byref(p))
        arch.call("cg_bc_apply", ctypes.byref(g), len(dims), vel, barr)
    return [f.to_numpy() for f in s.d["V"] + [s.d["P"]] + s.d["tau"]]


def ptdiff(arch, dims, calls):
    """C and q after the calls' iterations of one step (0: one iteration by its launches)."""
    nd, rng = len(dims), np.random.default_rng(9)
    grid = UniformGrid(origin=(-0.5,) * nd, extent=(1.0,) * nd, dims=dims, dtype=T)
    C, C_old, D = (Field(arch, grid, Center(), T) for _ in range(3))
    q = [Field(arch, grid, tuple(Vertex() if e == d else Center() for e in range(nd)), T) for d in range(nd)]
    C.from_numpy(rng.random(tuple(reversed(C.ext))))
    C_old.data.copy_(C.data)
    D.from_numpy(np.exp(rng.uniform(-1, 1, tuple(reversed(D.ext)))))
    s = _abi.cg_ptdiff_fields()
    s.C, s.C_old, s.D = C.desc(), C_old.desc(), D.desc()
    for k, f in enumerate(q):
        s.q[k] = f.desc()
    g, p = grid.desc(), ptdiff_params(grid, 1e-3, float(np.e))
    bc = to_cg_bc(nd, {"x": Dirichlet(0.0), "y": Neumann()} | ({"z": Neumann()} if nd == 3 else {}))
    start = C_old.data.clone()
    for n in calls:
        if n:
            arch.call("cg_ptdiff_run", ctypes.byref(g), ctypes.byref(s), ctypes.byref(p), ctypes.byref(bc), 1, n)
        else:
            arch.call("cg_ptdiff_update_q", ctypes.byref(g), ctypes.byref(s), ctypes.byref(p))
            arch.call("cg_ptdiff_update_C", ctypes.byref(g), ctypes.byref(s), ctypes.byref(p))
            arch.call("cg_bc_apply", ctypes.byref(g), 1, ctypes.byref(s.C), ctypes.byref(bc))
    assert (C_old.data == start).all() or len([n for n in calls if n]) > 1
    return [f.to_numpy() for f in [C] + q]


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


# (loop, sizes, iterations, whether the loop computes coefficients)
RULE = [(stokes, (60, 50), 4, False), (stokes, (60, 50), 5, True), (stokes, (16, 14, 12), 2, False), (stokes, (16, 14, 12), 3, True),
        (stokes, (220, 230), 2, True), (stokes, (220, 230), 1, False), (ptdiff, (120, 110), 24, False), (ptdiff, (20, 21, 22), 24, False),
        (ptdiff, (200, 210), 15, False), (ptdiff, (200, 210), 16, True), (ptdiff, (300, 270), 3, False), (ptdiff, (300, 270), 4, True)]


@pytest.mark.parametrize("loop,dims,n,coef", RULE)
def test_short_loops_on_small_grids_have_the_bits_of_their_launches(arch, loop, dims, n, coef):
    """Where filling the coefficients would cost more than it saves, a loop runs the kernels of the launches
    one by one and has their bits; elsewhere it differs from them by rounding: the per-launch tolerance times
    the launches."""
    a, b = loop(arch, dims, [n]), loop(arch, dims, [0] * n)
    assert _same(a, b) != coef
    for x, y in zip(a, b):
        assert np.max(np.abs(x - y)) <= rtol_for(T) * n * 10 * np.max(np.abs(y))


@pytest.mark.parametrize("loop,dims", [(stokes, (60, 50)), (stokes, (16, 14, 12)), (ptdiff, (40, 50)), (ptdiff, (20, 21, 22))])
def test_environment_decides(arch, monkeypatch, loop, dims):
    monkeypatch.setenv("CG_LOOP_COEF", "0")
    off, apart = loop(arch, dims, [20]), loop(arch, dims, [0] * 20)
    assert _same(off, apart)
    monkeypatch.setenv("CG_LOOP_COEF", "1")
    on = loop(arch, dims, [20])
    assert not _same(on, apart)
    for x, y in zip(on, apart):
        assert np.max(np.abs(x - y)) <= rtol_for(T) * 200 * np.max(np.abs(y))


@pytest.mark.parametrize("dims", [(2, 3), (41, 35), (300, 5), (5, 4, 3), (14, 12, 10)])
@pytest.mark.parametrize("kernels", ["ptdiff", "stokes"])
def test_block_shapes_of_the_loop_kernels(arch, monkeypatch, dims, kernels):
    """Every block shape, row by row and in order, gives the bits of 32 x 8 with the coefficients."""
    monkeypatch.setenv("CG_LOOP_COEF", "1")
    monkeypatch.setattr(shapes, "SHAPES", shapes.SHAPES + ["32x2", "64x1", "128x1", "256x1"])
    if kernels == "ptdiff":
        shapes.test_ptdiff_run_block_shapes(arch, monkeypatch, dims)
    else:
        shapes.test_stokes_pt_iterations_block_shapes(arch, monkeypatch, T, dims)
