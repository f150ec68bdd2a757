"""The rule by which a call takes scratch that it can do without (cg_scratch_spares)."""

import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "chmy.jl_gb300" / "csrc"
HARNESS = r"""
#include "cg_common.cuh"
int main() {
    const size_t G = (size_t)1 << 30;
    const size_t q[][3] = {{1, 0, 8}, {4, 0, 8}, {5, 0, 8}, {5, 2, 8}, {6, 2, 8}, {2, 2, 0}, {3, 2, 0}, {0, 0, 0}};
    for (auto& r : q) std::printf("%d ", (int)cg_scratch_spares(r[0] * G, r[1] * G, r[2] * G));
}
"""


def test_optional_scratch_leaves_as_much_free_as_it_takes(tmp_path):
    """(wanted, held by the slot, free): growth to at most half of what is free with the slot's own bytes
    given back; what the slot holds already is taken whatever is free."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no nvcc")
    src, exe = tmp_path / "h.cu", tmp_path / "h"
    src.write_text(HARNESS)
    subprocess.run([nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_103a,code=sm_103a", "-I", str(CSRC), "-o",
                    str(exe), str(src)], check=True, capture_output=True, text=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["1", "1", "0", "1", "0", "1", "0", "1"]
