"""Runs in which the caller passes one array for two fields: D = C (a diffusivity that follows the
solution), D = C_old (one that follows the last step) and C_old = C (no time term)."""

import ctypes

import numpy as np
import pytest

from _oracle import NpField, bc_apply, lib
from chmy_gb300 import _abi
from chmy_gb300.bcs import Neumann, to_cg_bc
from chmy_gb300.configs import ptdiff_params
from chmy_gb300.grids import Center, UniformGrid, Vertex
from gpu_helpers import assert_close, rtol_for, to_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [np.float64, np.float32])
@pytest.mark.parametrize("dims", [(21, 34), (33, 20, 18)])
@pytest.mark.parametrize("alias", ["D=C", "D=C_old", "C_old=C"])
@pytest.mark.parametrize("pitch", [0, 128])
def test_run_reads_the_array_of_the_moment(arch, T, dims, alias, pitch):
    """cg_ptdiff_run against the oracle's launches on the same aliased arrays: two steps of five
    iterations, per-launch tolerance times the launches."""
    nd = len(dims)
    grid = UniformGrid(origin=(T(-0.5),) * nd, extent=(T(1),) * nd, dims=dims, dtype=T)
    rng = np.random.default_rng(7)
    C, C_old, D = (NpField(grid, Center(), T) for _ in range(3))
    q = [NpField(grid, tuple(Vertex() if e == d else Center() for e in range(nd)), T) for d in range(nd)]
    for f in (C, C_old, D):
        f.a[...] = rng.uniform(0.5, 1.5, f.a.shape).astype(T)
    rows = dims[1] + 5 if pitch and nd == 3 else 0
    h = {"C": C, "C_old": C_old, "D": D}
    d = {k: to_gpu(arch, f, pitch, rows) for k, f in h.items()}
    qd = [to_gpu(arch, f, pitch, rows) for f in q]
    to, of = alias.split("=")
    h[to], d[to] = h[of], d[of]

    def desc(fs, qs):
        s = _abi.cg_ptdiff_fields()
        s.C, s.C_old, s.D = fs["C"].desc(), fs["C_old"].desc(), fs["D"].desc()
        for k, f in enumerate(qs):
            s.q[k] = f.desc()
        return s

    p = ptdiff_params(grid, dt=1e-3, Dmax=1.5)
    bc, g, hs = to_cg_bc(nd, Neumann()), grid.desc(), desc(h, q)
    arch.call("cg_ptdiff_run", ctypes.byref(g), ctypes.byref(desc(d, qd)), ctypes.byref(p), ctypes.byref(bc), 2, 5)
    for _ in range(2):
        h["C_old"].a[...] = h["C"].a
        for _ in range(5):
            lib().or_ptdiff_update_q(ctypes.byref(g), ctypes.byref(hs), ctypes.byref(p))
            lib().or_ptdiff_update_C(ctypes.byref(g), ctypes.byref(hs), ctypes.byref(p))
            bc_apply(grid, [h["C"]], [bc])
    for k in ("C", "C_old", "D"):
        assert_close(d[k], h[k], rtol_for(T) * 20, k)
    for a, b in zip(qd, q):
        assert_close(a, b, rtol_for(T) * 20, "q")
