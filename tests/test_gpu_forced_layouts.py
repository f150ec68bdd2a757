"""Layouts fixed by the environment are taken without timing the candidates."""

import os
import re
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
TESTS = Path(__file__).resolve().parent

HEAD = f"""
import ctypes, sys
sys.path[:0] = [{str(TESTS)!r}, {str(TESTS.parent / "chmy.jl_gb300")!r}]
import numpy as np
from chmy_gb300 import Arch, GB300Backend
arch = Arch(GB300Backend(), device_id=1)
"""


def tuned(script, **env):
    """The verbose lines of the autotuners while `script` runs in a process of its own."""
    base = {k: v for k, v in os.environ.items() if not k.startswith("CG_")} | {"CG_TUNE_VERBOSE": "1"} | env
    r = subprocess.run([sys.executable, "-c", HEAD + script], env=base, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
    return [l for l in r.stderr.splitlines() if " tune" in l]


@pytest.mark.parametrize("dims,layouts", [((31, 20, 17), ["0:0", "8:1", "0:4", "4:4"]), ((61, 40), ["0:0", "16:0", "0:1", "0:2", "0:3"])])
def test_march_layouts(arch, dims, layouts):
    script = f"from test_gpu_stokes import _pp_run, _bc_V\n_pp_run(arch, np.float32, {dims}, _bc_V({len(dims)}), 4)\n"
    name = f"march{len(dims)}d tune"
    assert any(name in l for l in tuned(script))
    for layout in layouts:
        assert not any(name in l for l in tuned(script, CG_MARCH_LAYOUT=layout)), layout


PTD = """
from chmy_gb300 import Field, _abi
from chmy_gb300.bcs import Neumann, Periodic, to_cg_bc
from chmy_gb300.configs import ptdiff_params
from chmy_gb300.grids import Center, UniformGrid, Vertex
T, dims = np.float32, (66, 40, 30)
grid = UniformGrid(origin=(T(-0.5),) * 3, extent=(T(1),) * 3, dims=dims, dtype=T)
C, C_old, D = (Field(arch, grid, Center(), T) for _ in range(3))
q = [Field(arch, grid, tuple(Vertex() if e == d else Center() for e in range(3)), T) for d in range(3)]
D.data.fill_(1.0)
s = _abi.cg_ptdiff_fields()
s.C, s.C_old, s.D = C.desc(), C_old.desc(), D.desc()
s.q = (_abi.cg_field * 3)(*[f.desc() for f in q])
p = ptdiff_params(grid, dt=1e-3, Dmax=1.0)
for spec in ({"x": Neumann(), "y": Neumann(), "z": Neumann()}, {"x": Periodic(), "y": Neumann(), "z": Neumann()}, None):
    print("--- tune", spec, file=sys.stderr, flush=True)
    bc = to_cg_bc(3, spec) if spec else None
    arch.call("cg_ptdiff_run", ctypes.byref(grid.desc()), ctypes.byref(s), ctypes.byref(p), ctypes.byref(bc) if bc else None, 1, 8)
"""


def test_ptdiff_layouts_are_timed_with_the_launches_of_the_run(arch):
    """Rules that the rows layouts fold, rules that they do not (a bc! launch follows every iteration) and
    no rules are three runs, each timed for itself: with the launch an iteration takes longer."""
    lines = tuned(PTD)
    runs, best = " ".join(lines).split("--- tune")[1:], []
    for log in runs:
        us = [float(w) for w in re.findall(r"seg \d+: ([\d.]+) us", log)]
        assert us, "a layout timed under other rules was taken"
        best.append(min(us))
    assert best[1] > best[0] + 1.0 and best[1] > best[2] + 1.0, best


PP2D = """
from test_gpu_stokes import _bc_V, _pp_run
from chmy_gb300.bcs import Neumann, Periodic, to_cg_bc
for bcs, niter in ((_bc_V(2), 6), ([to_cg_bc(2, {"x": Periodic(), "y": Neumann()}) for _ in range(2)], 6), (_bc_V(2), 2)):
    print("--- tune", file=sys.stderr, flush=True)
    _pp_run(arch, np.float32, (150, 131), bcs, niter)
"""


def test_tiles_are_timed_only_where_the_call_can_take_them(arch):
    """Ping-pong iterations whose rules fold, with periodic sides (a bc! launch between iterations), and two
    iterations: only the first can take the tile kernel. The others time the one-iteration kernel's segments
    and run the best of these."""
    runs = " ".join(tuned(PP2D)).split("--- tune")[1:]
    assert len(runs) == 3 and re.search(r"variant [123] ", runs[0])
    for log in runs[1:]:
        assert not re.search(r"variant [123] ", log) and (log is runs[2] or "variant 0 " in log)


DIFFUSION = """
from chmy_gb300 import Field
from chmy_gb300.grids import Center, UniformGrid
grid = UniformGrid(origin=(-1.0, -1.0), extent=(2.0, 2.0), dims=(700, 600))
A, B = (Field(arch, grid, Center()) for _ in range(2))
arch.call("cg_diffusion_run", ctypes.byref(grid.desc()), ctypes.byref(A.desc()), ctypes.byref(B.desc()), 1.0, 1e-6, None, 4)
"""


def test_diffusion_layouts(arch):
    assert any("diffusion step tune" in l for l in tuned(DIFFUSION))
    for layout in ("1:0", "8:1"):
        assert not tuned(DIFFUSION, CG_DIFFUSION_LAYOUT=layout)


DIFFUSION_BC = """
from chmy_gb300 import Field
from chmy_gb300.bcs import Neumann, to_cg_bc
from chmy_gb300.grids import Center, UniformGrid
grid = UniformGrid(origin=(-1.0, -1.0), extent=(2.0, 2.0), dims=(700, 610))
A, B = (Field(arch, grid, Center()) for _ in range(2))
for n in (8, 1):
    print("--- tune", file=sys.stderr, flush=True)
    arch.call("cg_diffusion_run", ctypes.byref(grid.desc()), ctypes.byref(A.desc()), ctypes.byref(B.desc()), 1.0, 1e-6,
              ctypes.byref(to_cg_bc(2, Neumann())), n)
"""


def test_one_diffusion_step_is_timed_as_an_ordinary_launch(arch):
    """Steps that follow each other can be dependent launches; a single step cannot, and takes a layout timed
    without."""
    runs = " ".join(tuned(DIFFUSION_BC)).split("--- tune")[1:]
    assert len(runs) == 2 and "dependent" in runs[0]
    assert "seg" in runs[1] and "dependent" not in runs[1]
