"""The time-step kernels of the shallow-ice runs (D_tile, H_tile) at the edges of their tiles."""

import ctypes

import numpy as np
import pytest

from _oracle import desc_array, lib
from gpu_helpers import assert_close, rtol_for, to_gpu
from test_gpu_sia import reference_params, setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [np.float32, np.float64])
@pytest.mark.parametrize("n", [(2, 2), (31, 8), (32, 9), (33, 16), (62, 7), (63, 33), (95, 24)])
@pytest.mark.parametrize("nsteps", [1, 6])
def test_run_at_tile_edges(arch, T, n, nsteps):
    """cg_sia_run against the oracle's loop, thickness and the last step's fluxes with all their
    boundary values: tiles of 32 and 31 columns by 8 rows, one cell more and one less; steps of both
    parities. Tolerances: per launch, times the steps."""
    grid, H, B, q = setup(T, n=n, seed=11)
    p = reference_params()
    Hg, Bg, qg = to_gpu(arch, H), to_gpu(arch, B), [to_gpu(arch, f) for f in q]
    g, dx, t_ref = grid.desc(), min(grid.spacing()), 0.0
    for _ in range(nsteps):
        dmax = ctypes.c_double()
        lib().or_sia_update_q(ctypes.byref(g), desc_array(q, 3), ctypes.byref(H.desc()), ctypes.byref(B.desc()), ctypes.byref(p),
                              ctypes.byref(dmax))
        dt = min(float(T(T(dx) * T(dx)) / T(dmax.value) / T(4.1)), 0.5)
        lib().or_sia_update_H(ctypes.byref(g), ctypes.byref(H.desc()), desc_array(q, 3), ctypes.byref(B.desc()), dt, ctypes.byref(p))
        t_ref += dt
    t = ctypes.c_double()
    arch.call("cg_sia_run", ctypes.byref(g), ctypes.byref(Hg.desc()), ctypes.byref(Bg.desc()), desc_array(qg, 3), ctypes.byref(p),
              nsteps, ctypes.byref(t))
    assert_close(Hg, H, rtol_for(T) * nsteps, "H")
    for a, b in zip(qg, q):
        assert_close(a, b, rtol_for(T) * nsteps * 10, "q")
    assert abs(t.value - t_ref) <= rtol_for(T) * nsteps * t_ref


@pytest.mark.parametrize("T", [np.float32, np.float64])
@pytest.mark.parametrize("n", [(2, 2), (2, 30), (28, 7), (29, 8), (30, 9), (31, 13), (59, 14), (88, 33), (200, 40)])
@pytest.mark.parametrize("glen", [3, 4])
def test_one_launch_per_step_has_the_bits_of_two(arch, monkeypatch, T, n, glen):
    """A step in one launch (tiles of 29 columns by 4, 8 or 13 rows that repeat their neighbours' cells)
    against D and the rest apart: thickness with its ghost layer, the last fluxes and the time, byte
    for byte, for runs of one step, of an even and of an odd number."""
    grid, H, B, q = setup(T, n=n, seed=7)
    p = reference_params()
    p.n = glen
    g = grid.desc()
    for nsteps in (1, 2, 7):
        out = {}
        for rows in ("0", "4", "8", "13", None):
            if rows is None:
                monkeypatch.delenv("CG_SIA_STEP_ROWS")
            else:
                monkeypatch.setenv("CG_SIA_STEP_ROWS", rows)
            Hg, Bg, qg = to_gpu(arch, H), to_gpu(arch, B), [to_gpu(arch, f) for f in q]
            t = ctypes.c_double()
            arch.call("cg_sia_run", ctypes.byref(g), ctypes.byref(Hg.desc()), ctypes.byref(Bg.desc()), desc_array(qg, 3),
                      ctypes.byref(p), nsteps, ctypes.byref(t))
            out[rows] = [f.to_numpy().tobytes() for f in [Hg] + qg] + [t.value]
        for rows in ("4", "8", "13", None):
            assert out[rows] == out["0"], (rows, nsteps)
