"""cg_diffusion_step at a size that no run has timed: its launch layout follows the size."""

import ctypes

import numpy as np
import pytest

from chmy_gb300 import Field
from chmy_gb300.grids import Center, UniformGrid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [np.float32, np.float64])
@pytest.mark.parametrize("n", [64, 128, 520])
def test_small_grids_take_short_segments(arch, monkeypatch, T, n):
    """A step is a chain over the rows of a segment, so a small grid with segments of 8 rows takes half as
    long again as with one, or twice as long. Untimed, a step is within a quarter of the best of one, two
    and four rows (the shortest of seven means over 60 steps)."""
    import torch

    grid = UniformGrid(origin=(T(-1),) * 2, extent=(T(2),) * 2, dims=(n + 1, n + 3), dtype=T)
    A, B = (Field(arch, grid, Center(), T) for _ in range(2))
    g, a, b = grid.desc(), A.desc(), B.desc()
    stream = torch.cuda.Stream()

    def took():
        best = 1e30
        for _ in range(7):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            torch.cuda._sleep(4_000_000)  # the host queues the steps behind it
            e[0].record()
            for _ in range(60):
                arch.call("cg_diffusion_step", ctypes.byref(g), ctypes.byref(b), ctypes.byref(a), 1.0, 1e-7, None)
            e[1].record()
            e[1].synchronize()
            best = min(best, e[0].elapsed_time(e[1]) / 60 * 1e3)
        return best

    try:
        with torch.cuda.stream(stream):
            arch.activate()  # the library works on torch's current stream
            untimed, forced = took(), []
            for seg in (1, 2, 4):
                monkeypatch.setenv("CG_DIFFUSION_LAYOUT", f"{seg}:0")
                forced.append(took())
    finally:
        arch.activate()
    assert untimed < 1.25 * min(forced), (untimed, forced)
