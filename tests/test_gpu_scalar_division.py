"""Divisions by the scalar-viscosity form's constants (ConstDiv) have the bits of the division."""

import ctypes

import numpy as np
import pytest

from _oracle import NpField
from chmy_gb300 import TensorField, VectorField, Field
from chmy_gb300.grids import Center, UniformGrid
from chmy_gb300.kernels import stokes_fields, stokes_params

pytestmark = pytest.mark.gpu


def _values(shape, rng):
    """Values over the whole exponent range, with zeros, subnormals, infinities and NaN among them."""
    x = rng.standard_normal(shape) * 2.0 ** rng.integers(-40, 40, shape)
    wide = rng.random(shape) < 0.3
    x[wide] *= 2.0 ** rng.integers(-980, 980, shape)[wide].astype(float)
    flat = x.reshape(-1)
    special = [0.0, -0.0, 5e-324, -5e-324, 1e-310, 1.7e308, -1.7e308, np.inf, -np.inf, np.nan, 2.0**-700, 2.0**700, 2.0**-701]
    flat[rng.choice(flat.size, 40 * len(special), replace=False)] = np.repeat(special, 40)
    return x


@pytest.mark.parametrize("c", [(0.37, 1.3, 0.011, 0.7), (1.0, 1.0, 1e-2, 3.0), (1e-70, 1.0, 1e70, 1e-65)])
def test_scalar_viscosity_divisions(arch, c):
    """update_stress! with V = 0, tau_old = 0 and eta_ve = dtau_r = 1 leaves tau + (-tau/(G dt) - tau/eta),
    and update_velocity! with tau = 0, V = 0 leaves (r nu_dtau)/eta_ve: every other operation is exact or
    rounds alone, so numpy's division gives the kernels' bits (constants inside and outside the range of
    the short form, arguments of every kind)."""
    eta, G, dt, eve = c
    grid = UniformGrid(origin=(0.0, 0.0), extent=(1.0, 1.0), dims=(64, 61))
    rng = np.random.default_rng(2)
    V, rV, tau, old = (k(arch, grid) for k in (VectorField, VectorField, TensorField, TensorField))
    P, div = Field(arch, grid, Center()), Field(arch, grid, Center())
    g = grid.desc()
    start = []
    for f in tau:
        f.from_numpy(_values(tuple(reversed(f.ext)), rng))
        start.append(f.to_numpy())
    s = stokes_fields(V=V, r_V=rV, P=P, divV=div, tau=tau, tau_old=old)
    arch.call("cg_stokes_update_stress", ctypes.byref(g), ctypes.byref(s),
              ctypes.byref(stokes_params(eta=eta, eta_ve=1.0, G=G, dt=dt, dtau_Pr=0.5, dtau_r=1.0)))
    for f, t in zip(tau, start):
        with np.errstate(all="ignore"):
            want = t + (-t / (G * dt) - t / eta)
        a, b = f.to_numpy()[1:64, 1:67], want[1:64, 1:67]  # logical 0 .. n+1
        assert np.array_equal(np.isnan(a), np.isnan(b))
        assert np.array_equal(a[~np.isnan(b)], b[~np.isnan(b)])
    for f in tau:
        f.data.zero_()
    p = NpField(grid, Center())
    p.a[...] = _values(p.a.shape, rng)
    P.from_numpy(p.a)
    nu = 0.31
    arch.call("cg_stokes_update_velocity", ctypes.byref(g), ctypes.byref(s), ctypes.byref(stokes_params(eta_ve=eve, nu_dtau=nu)))
    with np.errstate(all="ignore"):
        r = -((p.a[1:64, 1:67] - p.a[1:64, 0:66]) * g.inv_spacing[0])
        want = (r * nu) / eve
    a = V.x.to_numpy()[1:64, 1:67]
    ok = np.isfinite(r)
    assert np.array_equal(a[ok], want[ok])
