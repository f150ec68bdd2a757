"""The check of the defect-correction solve's inner loop (max |divV|, |r_V|, |r_tau| in one launch):
a residual that sits in the last interior row, at the sizes around its 32 x 8 blocks, has to be
seen, or the inner loop ends at its first check and the solve does not reach its tolerance."""

import dataclasses

import numpy as np
import pytest

from chmy_gb300 import _abi
from chmy_gb300.configs import stokes2d_inclusions, stokes3d_grf
from chmy_gb300.solvers import StokesSolver
from test_gpu_solve import _compare_states

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nd,n,last", [(2, 30, 0), (2, 31, 1), (2, 33, 0), (2, 62, 1), (3, 7, 0), (3, 15, 2), (3, 18, 1)])
def test_check_sees_the_last_interior_faces(arch, nd, n, last):
    pb = stokes2d_inclusions(n, ncheck=16) if nd == 2 else stokes3d_grf(n, ncheck=16)
    host = dict(pb.host)
    rho = [None] * nd
    # the padded index of face n, the last whose momentum residual counts, is n + 1 along each dim
    rho[last] = np.zeros_like(pb.host["V"][last])
    rho[last][(n + 1,) * nd] = 1.0
    host["rho_g"] = rho
    pb = dataclasses.replace(pb, host=host)
    ref, dc = StokesSolver(arch, pb), StokesSolver(arch, pb)
    for s in (ref, dc):
        s.apply_bc()
    r64 = ref.solve(precision=_abi.CG_F64)
    r32 = dc.solve(precision=_abi.CG_F32, max_outer=8, inner_rtol=1e-5)
    assert r64.converged == 1 and r32.converged == 1, (r64.iterations, r32.outer, r32.iterations, list(r32.err))
    assert r32.outer <= 4
    _compare_states(ref, dc, nd)
