"""A thermal loop whose viscosity is the temperature's array."""

import ctypes

import numpy as np
import pytest

from chmy_gb300 import _abi
from chmy_gb300.bcs import Neumann, to_cg_bc
from gpu_helpers import rtol_for, to_gpu
from test_gpu_stokes import StokesSet, _bc_V, pt_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(33, 21), (9, 10, 8)])
@pytest.mark.parametrize("which", ["eta", "inv_eta"])
def test_viscosity_follows_the_array(arch, dims, which):
    """cg_stokes_pt_iterations_thermal with eta (or 1/eta) = T against its launches one by one. T alternates
    with a second buffer, so the array holds iteration 0's T during iterations 0 and 1, iteration 2's
    during 2 and 3. Per-launch tolerance times the launches, as the loop's kernels contract otherwise."""
    T, nd, niter = np.float64, len(dims), 4
    loop, ref = (StokesSet(arch, dims, T, 61, False, thermal=True) for _ in range(2))
    for s in (loop, ref):
        rng = np.random.default_rng(3)
        for k in ("T", "T_old"):
            a = (1.0 + 0.2 * rng.random(s.h[k].a.shape)).astype(T)
            s.d[k].from_numpy(a)
        s.d[which] = s.d["T"]
    bcs, bcT = (_abi.cg_bc * 3)(*_bc_V(nd)), to_cg_bc(nd, Neumann())
    g, p = loop.grid.desc(), pt_params(loop.grid, True)
    arch.call("cg_stokes_pt_iterations_thermal", ctypes.byref(g), ctypes.byref(loop.dev_desc()), ctypes.byref(p), bcs,
              ctypes.byref(bcT), niter)
    A, B = ref.d["T"], to_gpu(arch, ref.h["T"])
    B.data.copy_(A.data)
    vel = (_abi.cg_field * 3)(*[f.desc() for f in ref.d["V"]])
    for it in range(niter):
        ref.d["T"], out = (A, B) if it % 2 == 0 else (B, A)
        d = ref.dev_desc()
        arch.call("cg_stokes_update_stress", ctypes.byref(g), ctypes.byref(d), ctypes.byref(p))
        arch.call("cg_stokes_update_velocity", ctypes.byref(g), ctypes.byref(d), ctypes.byref(p))
        arch.call("cg_bc_apply", ctypes.byref(g), nd, vel, bcs)
        arch.call("cg_stokes_thermal_step", ctypes.byref(g), ctypes.byref(d), ctypes.byref(p), ctypes.byref(bcT), ctypes.byref(out.desc()))
    ref.d["T"] = A
    for k in ("V", "P", "tau", "T"):
        for a, b in zip(*[s.d[k] if isinstance(s.d[k], list) else [s.d[k]] for s in (loop, ref)]):
            if a is None:
                continue
            x, y = a.to_numpy(), b.to_numpy()
            assert np.max(np.abs(x - y)) <= rtol_for(T) * niter * 10 * np.max(np.abs(y)), k
