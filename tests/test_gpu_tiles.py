"""The 2D Stokes tile kernel (march2d_tile_kernel: several PT iterations per launch) in Chmy's dense
layout, forced with CG_MARCH_LAYOUT=0:<variant>, at the edges of its tiles."""

import ctypes

import numpy as np
import pytest

from _oracle import stokes_desc
from gpu_helpers import assert_close, to_gpu
from test_gpu_stokes import _bc_mix, _pp_run

pytestmark = pytest.mark.gpu
T = np.float32


@pytest.mark.parametrize("variant", [1, 2, 3])
@pytest.mark.parametrize("kind", ["neumann_vertex", "mixed"])
@pytest.mark.parametrize("dims", [(2, 2), (28, 60), (29, 61), (52, 27), (53, 109), (76, 77), (100, 33)])
@pytest.mark.parametrize("niter", [4, 18])
def test_tiles_match_oracle(arch, monkeypatch, variant, kind, dims, niter):
    """Both buffers after niter and niter - 1 iterations equal the oracle's bit for bit: grids that
    fill one tile, exceed it by a column or row, and end inside a halo (tiles are 32 columns by 32 or
    64 rows, with 4 or 8 rings of halo); chunks that divide evenly and that leave a remainder."""
    monkeypatch.setenv("CG_MARCH_LAYOUT", f"0:{variant}")
    s, partner, prev, _ = _pp_run(arch, T, dims, _bc_mix(kind), niter, seed=61)
    for name in ("V", "P", "tau", "divV", "r_V"):
        hv = s.h[name] if isinstance(s.h[name], list) else [s.h[name]]
        dv = s.d[name] if isinstance(s.d[name], list) else [s.d[name]]
        for a, b in zip(dv, hv):
            if b is not None:
                assert_close(a, b, 0.0, f"tiles {variant} {kind} {name}", exact=True)
    for a, b in zip(partner["V"], prev):
        assert np.array_equal(a.to_numpy().view(np.uint8), b.view(np.uint8))


@pytest.mark.parametrize("variant", [1, 2, 3])
@pytest.mark.parametrize("with_bc", [False, True])
def test_tiles_with_buffers_that_differ_outside_the_launch_range(arch, monkeypatch, variant, with_bc):
    """The partner buffers hold other values outside [0, n+1]^2: iterations read them in turn, and the
    tile kernel leaves the bits of the one-iteration kernel."""
    out = []
    for layout in ("0:0", f"0:{variant}"):
        monkeypatch.setenv("CG_MARCH_LAYOUT", layout)
        s, partner, _, (g, da, _, p, barr) = _pp_run(arch, T, (57, 70), _bc_mix("mixed"), 2, seed=67)
        rng = np.random.default_rng(5)
        other = {}
        for k in ("V", "P", "tau"):
            fs = s.h[k] if isinstance(s.h[k], list) else [s.h[k]]
            devs = []
            for f in fs:
                d = to_gpu(arch, f)
                a = f.a.copy()
                ring = rng.standard_normal(a.shape).astype(T)
                keep = np.zeros(a.shape, bool)
                keep[1:1 + 72, 1:1 + 59] = True  # logical 0 .. n+1
                a[~keep] = ring[~keep]
                d.from_numpy(a)
                devs.append(d)
            other[k] = devs if isinstance(s.h[k], list) else devs[0]
        db = stokes_desc(V=other["V"], P=other["P"], tau=other["tau"])
        bc = barr if with_bc else None
        arch.call("cg_stokes_pt_iterations_pp", ctypes.byref(g), ctypes.byref(da), ctypes.byref(db), ctypes.byref(p), bc, 14)
        arch.synchronize()
        out.append([f.to_numpy() for k in ("V", "tau", "r_V") for f in s.d[k]] + [s.d["P"].to_numpy(), s.d["divV"].to_numpy()]
                   + [f.to_numpy() for f in other["V"] + other["tau"]])
    for a, b in zip(*out):
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))


@pytest.mark.parametrize("layout", ["0:4", "4:4", "5:1", "8:0"])
@pytest.mark.parametrize("dims", [(31, 20, 70), (13, 12, 11), (61, 7, 5)])
@pytest.mark.parametrize("pitch", [0, 512])
def test_3d_layouts_match_oracle(arch, monkeypatch, layout, dims, pitch):
    """The 3D march with 122 registers and with short z segments (CG_MARCH_LAYOUT=<segment>:<variant>),
    in the dense layout (class strides) and in one with shared strides: the oracle's bits."""
    from test_gpu_stokes import _bc_V

    monkeypatch.setenv("CG_MARCH_LAYOUT", layout)
    rows = dims[1] + 5 if pitch else 0
    s, _, _, _ = _pp_run(arch, T, dims, _bc_V(3), 4, seed=71, pitch_align=pitch, plane_rows=rows)
    for name in ("V", "P", "tau", "divV", "r_V"):
        hv = s.h[name] if isinstance(s.h[name], list) else [s.h[name]]
        dv = s.d[name] if isinstance(s.d[name], list) else [s.d[name]]
        for a, b in zip(dv, hv):
            if b is not None:
                assert_close(a, b, 0.0, f"3d {layout} {name}", exact=True)
