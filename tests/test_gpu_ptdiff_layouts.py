"""The layout that cg_ptdiff_run caches for a 3D FP32 run belongs to the strides it was timed with: the
same grid and pitch with other plane heights of q must not run it."""

import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import ctypes, sys
sys.path[:0] = [{tests!r}, {pkg!r}]
import numpy as np
from _oracle import NpField, bc_apply, lib
from chmy_gb300 import Arch, GB300Backend, _abi
from chmy_gb300.bcs import Neumann, to_cg_bc
from chmy_gb300.configs import ptdiff_params
from chmy_gb300.grids import Center, UniformGrid, Vertex
from gpu_helpers import assert_close, random_field, to_gpu

T, dims = np.float32, (33, 20, 18)
arch = Arch(GB300Backend(), device_id=1)
grid = UniformGrid(origin=(T(-0.5),) * 3, extent=(T(1),) * 3, dims=dims, dtype=T)
g, bc = grid.desc(), to_cg_bc(3, Neumann())


def desc(fs):
    s = _abi.cg_ptdiff_fields()
    s.C, s.C_old, s.D = fs["C"].desc(), fs["C_old"].desc(), fs["D"].desc()
    s.q = (_abi.cg_field * 3)(*[f.desc() for f in fs["q"]])
    return s


rows = dims[1] + 5
for qx, qy in ((rows, rows), (rows + 3, rows), (rows, rows + 4)):
    rng = np.random.default_rng(5)
    h = {{"C": random_field(grid, Center(), T, rng), "C_old": NpField(grid, Center(), T), "D": NpField(grid, Center(), T),
         "q": [random_field(grid, tuple(Vertex() if e == d else Center() for e in range(3)), T, rng, 0.1) for d in range(3)]}}
    h["D"].a[...] = np.exp(rng.uniform(-1, 1, h["D"].a.shape)).astype(T)
    d = {{k: to_gpu(arch, h[k], 128, rows) for k in ("C", "C_old", "D")}}
    d["q"] = [to_gpu(arch, f, 128, r) for f, r in zip(h["q"], (qx, qy, rows))]
    p, hs = ptdiff_params(grid, dt=1e-3, Dmax=float(h["D"].a.max())), desc(h)
    print("run", qx, qy, file=sys.stderr, flush=True)
    arch.call("cg_ptdiff_run", ctypes.byref(g), ctypes.byref(desc(d)), ctypes.byref(p), ctypes.byref(bc), 1, 6)
    h["C_old"].a[...] = h["C"].a
    for _ in range(6):
        lib().or_ptdiff_update_q(ctypes.byref(g), ctypes.byref(hs), ctypes.byref(p))
        lib().or_ptdiff_update_C(ctypes.byref(g), ctypes.byref(hs), ctypes.byref(p))
        bc_apply(grid, [h["C"]], [bc])
    assert_close(d["C"], h["C"], 0.0, "C", exact=True)
    for a, b in zip(d["q"], h["q"]):
        assert_close(a, b, 0.0, "q", exact=True)
"""


def test_plane_heights_of_q_are_part_of_the_cached_layout(arch):
    """Three runs of one size and pitch in one process: C, D and q of one plane height, then q.x, then
    q.y of another. Each is timed for itself, and each equals the oracle bit for bit."""
    tests = Path(__file__).resolve().parent
    src = SCRIPT.format(tests=str(tests), pkg=str(tests.parent / "chmy.jl_gb300"))
    env = {k: v for k, v in os.environ.items() if not k.startswith("CG_")} | {"CG_TUNE_VERBOSE": "1"}
    r = subprocess.run([sys.executable, "-c", src], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
    runs = r.stderr.split("run ")[1:]
    assert len(runs) == 3
    for k, log in enumerate(runs):
        assert "ptdiff3d tune 33x20x18" in log, f"run {k} took the layout cached by an earlier one"
