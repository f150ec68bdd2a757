"""The thermal step sharing a launch with the next iteration's update_stress!, and bc!(T) with the next
bc!(V), against the kernels apart (CG_BLOCK keeps them apart)."""

import ctypes

import numpy as np
import pytest

from chmy_gb300 import _abi
from chmy_gb300.bcs import Neumann, to_cg_bc
from test_gpu_stokes import StokesSet, _bc_V, pt_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [np.float32, np.float64])
@pytest.mark.parametrize("var_eta", [False, True])
@pytest.mark.parametrize("dims", [(2, 2), (29, 6), (30, 7), (31, 10), (61, 33)])
@pytest.mark.parametrize("with_bc", [True, False])
def test_pairs_have_the_bits_of_the_kernels_apart(arch, monkeypatch, T, var_eta, dims, with_bc):
    """Edges of the 32 x 4 stress blocks and the 31 x 4 thermal tiles, the loop's coefficients (variable
    viscosity, from four iterations on) and the plain form; no iteration paired, one, an even and an
    odd number; with and without conditions on V."""
    bcs = (_abi.cg_bc * 3)(*_bc_V(2))
    bcT = to_cg_bc(2, {"x": Neumann(), "y": Neumann()})
    for niter in (1, 2, 5):
        out = []
        for apart in (False, True):
            monkeypatch.setenv("CG_BLOCK", "32x8" if apart else "")
            s = StokesSet(arch, dims, T, 61, var_eta, thermal=True)
            p = pt_params(s.grid, var_eta)
            g = s.grid.desc()
            arch.call("cg_stokes_pt_iterations_thermal", ctypes.byref(g), ctypes.byref(s.dev_desc()), ctypes.byref(p),
                      bcs if with_bc else None, ctypes.byref(bcT), niter)
            fields = [f for v in s.d.values() for f in (v if isinstance(v, list) else [v]) if f is not None]
            out.append([f.to_numpy().tobytes() for f in fields])
        assert out[0] == out[1], niter
