"""Layouts fixed by the environment are taken without timing the candidates."""

import os
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
