"""Calls whose scratch finds no room. CG_SCRATCH_LIMIT fails a scratch request as an allocation on a
full device does."""

import ctypes

import numpy as np
import pytest

from _oracle import NpField, bc_apply, lib
from chmy_gb300 import _abi
from chmy_gb300.bcs import Dirichlet, Neumann, to_cg_bc
from chmy_gb300.configs import ptdiff_params
from chmy_gb300.grids import Center, UniformGrid, Vertex
from gpu_helpers import assert_close, random_field, rtol_for, to_gpu

pytestmark = pytest.mark.gpu
SMALL = "4096"  # room for flags and words, for no field


def _pd_desc(fs):
    s = _abi.cg_ptdiff_fields()
    s.C, s.C_old, s.D = fs["C"].desc(), fs["C_old"].desc(), fs["D"].desc()
    s.q = (_abi.cg_field * 3)(*[f.desc() for f in fs["q"]])
    return s


@pytest.mark.parametrize("T", [np.float32, np.float64])
@pytest.mark.parametrize("pitch", [0, 128])
@pytest.mark.parametrize("npt", [5, 6])
def test_ptdiff_run_without_room(arch, monkeypatch, T, pitch, npt):
    """cg_ptdiff_run without its partner buffers (FP32) or coefficients (FP64) runs in place: two steps
    against the oracle, per-launch tolerance times the launches."""
    monkeypatch.setenv("CG_SCRATCH_LIMIT", SMALL)
    dims = (33, 20, 18)
    grid = UniformGrid(origin=(T(-0.5),) * 3, extent=(T(1),) * 3, dims=dims, dtype=T)
    rng = np.random.default_rng(5)
    h = {"C": random_field(grid, Center(), T, rng), "C_old": NpField(grid, Center(), T), "D": NpField(grid, Center(), T),
         "q": [random_field(grid, tuple(Vertex() if e == d else Center() for e in range(3)), T, rng, 0.1) for d in range(3)]}
    h["D"].a[...] = np.exp(rng.uniform(-1, 1, h["D"].a.shape)).astype(T)
    rows = dims[1] + 5 if pitch else 0
    d = {k: ([to_gpu(arch, f, pitch, rows) for f in v] if isinstance(v, list) else to_gpu(arch, v, pitch, rows)) for k, v in h.items()}
    p = ptdiff_params(grid, dt=1e-3, Dmax=float(h["D"].a.max()))
    bc = to_cg_bc(3, {"x": Dirichlet(0.2), "y": Neumann(), "z": Neumann(0.1)})
    g, hs = grid.desc(), _pd_desc(h)
    arch.call("cg_ptdiff_run", ctypes.byref(g), ctypes.byref(_pd_desc(d)), ctypes.byref(p), ctypes.byref(bc), 2, npt)
    for _ in range(2):
        h["C_old"].a[...] = h["C"].a
        for _ in range(npt):
            lib().or_ptdiff_update_q(ctypes.byref(g), ctypes.byref(hs), ctypes.byref(p))
            lib().or_ptdiff_update_C(ctypes.byref(g), ctypes.byref(hs), ctypes.byref(p))
            bc_apply(grid, [h["C"]], [bc])
    for k in ("C", "C_old"):
        assert_close(d[k], h[k], rtol_for(T) * 2 * npt, k)
    for a, b in zip(d["q"], h["q"]):
        assert_close(a, b, rtol_for(T) * 2 * npt, "q")


@pytest.mark.parametrize("dims", [(60, 50), (16, 14, 12)])
def test_stokes_loop_without_room(arch, monkeypatch, dims):
    """An FP64 loop without its viscosity terms has the bits of its launches one by one."""
    from test_gpu_loop_coef import stokes

    monkeypatch.setenv("CG_SCRATCH_LIMIT", SMALL)
    for a, b in zip(stokes(arch, dims, [20]), stokes(arch, dims, [0] * 20)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("T", [np.float32, np.float64])
def test_sia_run_without_room_for_second_buffers(arch, monkeypatch, T):
    """Three arrays of scratch instead of five: two launches a step, the same bits; one array less is an
    error that says so."""
    from chmy_gb300 import ChmyError
    from test_gpu_sia import reference_params, setup
    from _oracle import desc_array

    grid, H, B, q = setup(T, n=(66, 41), seed=7)
    p, out = reference_params(), []
    array = H.a.nbytes + 255 & ~255
    for limit in (None, 4 * array):
        if limit:
            monkeypatch.setenv("CG_SCRATCH_LIMIT", str(limit))
        Hg, Bg, qg = to_gpu(arch, H), to_gpu(arch, B), [to_gpu(arch, f) for f in q]
        g, t = grid.desc(), ctypes.c_double()
        call = lambda: arch.call("cg_sia_run", ctypes.byref(g), ctypes.byref(Hg.desc()), ctypes.byref(Bg.desc()), desc_array(qg, 3),
                                 ctypes.byref(p), 7, ctypes.byref(t))
        call()
        out.append([f.to_numpy().tobytes() for f in [Hg] + qg] + [t.value])
    assert out[0] == out[1]
    monkeypatch.setenv("CG_SCRATCH_LIMIT", str(2 * array))
    with pytest.raises(ChmyError, match="scratch"):
        call()
