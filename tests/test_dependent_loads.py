"""Loads of the kernels that are launched as dependent ones. Such a kernel is resident while the launch
before it still writes its outputs, so what a chain of launches writes may not be read by `__ldg`
(a non-coherent load is only defined for data that does not change while the kernel runs)."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "chmy.jl_gb300" / "csrc"
# what no launch of an iteration chain writes, by the names the kernels give it
CONSTANT = re.compile(r"f\.(?:ieta|t\w\w_o|tau_o\[\d\]|fP|rho[xy]|rho\[\d\]|D|Co)(?!\w)")


def _code(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def _call_args(text, call):
    """The text of the arguments of every `call(`."""
    for m in re.finditer(re.escape(call) + r"\(", text):
        depth, k = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[k], 0)
            k += 1
        yield text[m.end() : k - 1]


@pytest.mark.parametrize("name", ["cg_stokes_kernels.cuh", "cg_march3d.cuh", "cg_march2d_tile.cuh"])
def test_marching_kernels_read_the_state_by_plain_loads(name):
    text = _code(name)
    for args in _call_args(text, ".ldc"):
        assert CONSTANT.search(args), f"{name}: ldc({args})"
    # __ldg appears in the accessor of constant inputs alone
    for m in re.finditer("__ldg", text):
        head = text.rfind("__device__", 0, m.start())
        assert " ldc(" in text[head : m.start()], f"{name}: {text[m.start() : m.start() + 60]}"


def test_pt_diffusion_rows_kernel_reads_C_and_q_by_plain_loads():
    text = _code("cg_ptdiff.cu")
    body = text[text.index("ptd_rows_kernel(const PDM<T> f") : text.index("bool pd_edges(")]
    calls = list(_call_args(body, "__ldg"))
    assert calls
    for args in calls:
        assert CONSTANT.search(args), f"ptd_rows_kernel: __ldg({args})"
    # the kernels that read C and q by __ldg are launched the ordinary way
    assert re.search(r"ptd_march3d_kernel<[^;]*><<<", text) and not re.search(r"cg_launch\(\s*ptd_march3d_kernel", text)
