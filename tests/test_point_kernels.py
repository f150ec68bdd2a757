"""Host-side and source rules of the per-point kernels (cg_common.cuh's launch_point and point_grid)."""

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "chmy.jl_gb300" / "csrc"


def _code(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def test_the_order_of_points_is_no_branch_in_a_kernel():
    """Whether a block takes its points row by row or in order is a template parameter: as a branch on the
    block's shape it cost the FP32 kernels, which memory bounds, up to a third."""
    text = _code("cg_common.cuh")
    i = text.index("bool launch_point(")
    assert not re.search(r"blockDim\.[xy]\s*[=!<>]=?\s*\d", text[i : text.index("\n}\n", i)])
    for name in ("cg_stokes_kernels.cuh", "cg_ptdiff.cu"):
        calls = re.findall(r"launch_point<([^>]*)>", _code(name))
        assert calls and all(c in ("ND, FLAT", "ND, true") for c in calls), (name, calls)
