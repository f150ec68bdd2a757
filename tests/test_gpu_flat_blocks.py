"""Blocks of one row of threads (CG_BLOCK=<x>x1) take a plane's points in order instead of row by row:
the bits of the 32 x 8 shape, for x extents shorter and longer than a block and for planes that end
inside one."""

import numpy as np
import pytest

import test_gpu_block_shapes as shapes

pytestmark = pytest.mark.gpu
FLAT = ["64x1", "128x1", "256x1"]


@pytest.mark.parametrize("T", [np.float32, np.float64])
@pytest.mark.parametrize("dims", [(2, 3), (37, 29), (62, 6), (300, 5), (5, 4, 3), (13, 12, 11), (63, 2, 3)])
def test_stokes_loops(arch, monkeypatch, T, dims):
    monkeypatch.setattr(shapes, "SHAPES", FLAT)
    shapes.test_stokes_pt_iterations_block_shapes(arch, monkeypatch, T, dims)


@pytest.mark.parametrize("dims", [(2, 3), (41, 35), (62, 6), (300, 5), (5, 4, 3), (14, 12, 10), (63, 2, 3)])
def test_ptdiff_loops(arch, monkeypatch, dims):
    monkeypatch.setattr(shapes, "SHAPES", FLAT)
    shapes.test_ptdiff_run_block_shapes(arch, monkeypatch, dims)
