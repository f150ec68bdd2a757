"""Defect-correction solves of one grid, parameters and ncheck with other kinds of conditions: the second
one applies its own rules, not those of the first one's captured chunk."""

import dataclasses

import numpy as np
import pytest

from chmy_gb300 import Arch, GB300Backend, _abi
from chmy_gb300.bcs import Dirichlet, Neumann, to_cg_bc
from chmy_gb300.configs import stokes2d_inclusions, stokes3d_grf
from chmy_gb300.solvers import StokesSolver

pytestmark = pytest.mark.gpu


def _no_slip(nd):
    return [to_cg_bc(nd, {"xyz"[e]: Dirichlet() for e in range(nd)}) for _ in range(nd)]


def _free_slip(nd):
    return [to_cg_bc(nd, {"xyz"[e]: Dirichlet() if e == d else Neumann() for e in range(nd)}) for d in range(nd)]


@pytest.mark.parametrize("nd", [2, 3])
def test_second_solve_applies_its_own_rules(arch, nd):
    """A free-slip solve, then a no-slip one in the same context, against the no-slip solve in a new
    context: the same iterations and the same bits."""
    pb = stokes2d_inclusions(40, ncheck=20) if nd == 2 else stokes3d_grf(14, ncheck=20)
    host = dict(pb.host)
    rho = [None] * nd
    rho[nd - 1] = np.zeros_like(pb.host["V"][nd - 1])
    rho[nd - 1][tuple(slice(m // 3, m // 2) for m in rho[nd - 1].shape)] = 1.0
    host["rho_g"] = rho
    host["V"] = [np.zeros_like(a) for a in pb.host["V"]]
    slip = dataclasses.replace(pb, host=host, bc_V=_free_slip(nd))
    stick = dataclasses.replace(pb, host=host, bc_V=_no_slip(nd))

    def solve(a, problem):
        s = StokesSolver(a, problem)
        s.apply_bc()
        r = s.solve(precision=_abi.CG_F32, max_outer=8, inner_rtol=1e-5)
        assert r.converged == 1, (r.iterations, r.outer)
        return r.iterations, [f.to_numpy() for f in s.fields["V"] + s.fields["tau"]]

    solve(arch, slip)
    got = solve(arch, stick)
    other = Arch(GB300Backend(), device_id=1)
    want = solve(other, stick)
    other.close()
    assert got[0] == want[0]
    for a, b in zip(got[1], want[1]):
        assert np.array_equal(a, b)
