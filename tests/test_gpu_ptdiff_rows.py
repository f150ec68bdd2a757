"""The PT-diffusion iteration with several rows per thread (ptd_rows_kernel, layouts 8 to 10) with
bc! folded into its stores, in the pool layout and in Chmy's dense layout."""

import ctypes

import numpy as np
import pytest

from _oracle import NpField, bc_apply, lib
from chmy_gb300 import _abi
from chmy_gb300.bcs import Dirichlet, Neumann, Periodic, to_cg_bc
from chmy_gb300.configs import ptdiff_params
from chmy_gb300.grids import Center, UniformGrid, Vertex
from gpu_helpers import assert_close, random_field, to_gpu

pytestmark = pytest.mark.gpu
T = np.float32
C_, V_ = Center(), Vertex()
SPECS = {
    "mixed": {"x": (Dirichlet(0.2), Neumann(-0.1)), "y": (Neumann(0.3), Dirichlet(0.1)), "z": (Neumann(), Dirichlet(-0.2))},
    "one_sided": {"x": (None, Dirichlet(0.3)), "y": (Neumann(0.1), None), "z": None},
    "periodic_z": {"x": Neumann(), "y": Dirichlet(0.1), "z": Periodic()},
    "none": None,
}


def _desc(fs):
    s = _abi.cg_ptdiff_fields()
    s.C, s.C_old, s.D = fs["C"].desc(), fs["C_old"].desc(), fs["D"].desc()
    s.q = (_abi.cg_field * 3)(*[f.desc() for f in fs["q"]])
    return s


@pytest.mark.parametrize("variant", [8, 9, 10])
@pytest.mark.parametrize("pitch", [0, 128])
@pytest.mark.parametrize("dims", [(2, 2, 2), (28, 3, 5), (29, 6, 4), (31, 7, 17), (58, 9, 3), (59, 2, 35)])
@pytest.mark.parametrize("kind", list(SPECS))
@pytest.mark.parametrize("npt", [1, 4])
def test_rows_equal_oracle(arch, monkeypatch, variant, pitch, dims, kind, npt):
    """cg_ptdiff_run equals the oracle bit for bit: strips of 30 columns filled, exceeded by one and
    cut short, 2 and 3 rows per thread with a remainder, z segments; every rule mix, and rules that
    are not folded; an odd count ends in the partner buffers."""
    monkeypatch.setenv("CG_PTD_VARIANT", str(variant))
    grid = UniformGrid(origin=(T(-0.5),) * 3, extent=(T(1), T(0.9), T(1.2)), dims=dims, dtype=T)
    rng = np.random.default_rng(17)
    h = {"C": random_field(grid, C_, T, rng), "C_old": NpField(grid, C_, T), "D": NpField(grid, C_, T),
         "q": [random_field(grid, tuple(V_ if e == d else C_ for e in range(3)), T, rng, 0.1) for d in range(3)]}
    h["D"].a[...] = np.exp(rng.uniform(-1, 1, h["D"].a.shape)).astype(T)
    rows = dims[1] + 5 if pitch else 0
    d = {k: ([to_gpu(arch, f, pitch, rows) for f in v] if isinstance(v, list) else to_gpu(arch, v, pitch, rows)) for k, v in h.items()}
    p = ptdiff_params(grid, dt=1e-3, Dmax=float(h["D"].a.max()))
    bc = to_cg_bc(3, SPECS[kind]) if kind != "none" else None
    g = grid.desc()
    hs = _desc(h)
    for _ in range(2):
        h["C_old"].a[...] = h["C"].a
        for _ in range(npt):
            lib().or_ptdiff_update_q(ctypes.byref(g), ctypes.byref(hs), ctypes.byref(p))
            lib().or_ptdiff_update_C(ctypes.byref(g), ctypes.byref(hs), ctypes.byref(p))
            if bc is not None:
                bc_apply(grid, [h["C"]], [bc])
    arch.call("cg_ptdiff_run", ctypes.byref(g), ctypes.byref(_desc(d)), ctypes.byref(p), ctypes.byref(bc) if bc is not None else None,
              2, npt)
    for k in ("C", "C_old"):
        assert_close(d[k], h[k], 0.0, k, exact=True)
    for a, b in zip(d["q"], h["q"]):
        assert_close(a, b, 0.0, "q", exact=True)
