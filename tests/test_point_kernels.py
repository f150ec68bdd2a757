"""Host-side and source rules of the per-point kernels (cg_common.cuh's launch_point and point_grid)."""

import re
import shutil
import subprocess
from pathlib import Path

import pytest

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


HARNESS = r"""
#include "cg_common.cuh"
#include <cstdlib>
int main(int argc, char** argv) {
    const int n[3] = {std::atoi(argv[1]), std::atoi(argv[2]), std::atoi(argv[3])};
    const dim3 block(std::atoi(argv[4]), std::atoi(argv[5]));
    const dim3 a = cgk::point_grid<2>(n, block), b = cgk::point_grid<3>(n, block);
    std::printf("%d %u %u %u %u %u\n", (int)cgk::in_order<2>(n, block), a.x, a.y, b.x, b.y, b.z);
}
"""


def test_every_point_of_a_plane_has_a_thread(tmp_path):
    """The grids of the per-point kernels: blocks of one row take the points in order only where an int counts
    the plane's points (a 65534^2 plane has 2^32), and then, as row by row, every point has one thread."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no nvcc")
    src = tmp_path / "h.cu"
    src.write_text(HARNESS)
    exe = tmp_path / "h"
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_103a,code=sm_103a", "-I", str(CSRC), "-o",
                    str(exe), str(src)], check=True, capture_output=True, text=True)
    for n0, n1 in ((5, 3), (95, 80), (46338, 46337), (46339, 46338), (65534, 65534), (200000, 30000), (1, 400000)):
        for bx, by in ((64, 1), (256, 1), (32, 8), (128, 2)):
            out = subprocess.run([str(exe), str(n0), str(n1), "7", str(bx), str(by)], check=True, capture_output=True, text=True).stdout
            order, ax, ay, cx, cy, cz = map(int, out.split())
            w, h = n0 + 2, n1 + 2
            assert order == (by == 1 and w * h <= 2**31 - 1 - 1024)
            assert (cx, cy, cz) == (ax, ay, 9)
            if order:
                assert ay == 1 and w * h <= ax * bx < 2**31
            else:
                assert (ax, ay) == (-(-w // bx), -(-h // by))


def test_large_layouts_keep_their_shared_strides():
    """Views whose offsets need 64 bits run the marching kernels with the layout that their strides have: with
    every array's own strides a 2D iteration took 15 % longer."""
    for name, launch in (("cg_stokes_kernels.cuh", "launch_march2d_ix"), ("cg_march3d.cuh", "launch_march3d_ix")):
        layouts = re.findall(launch + r"<T, long, (\w+),", _code(name))
        assert "kLayOwn" in layouts and "kLayLoc" in layouts, (name, layouts)
