"""1D blocks whose faces exchange fewer halo points than the stencil reaches: the points beyond the
exchange depth keep what the caller put there, on the resident path as on the others.  Against the C
oracle: FP64 1e-12 of the largest value per variable, FP32 1e-5, as for deeper exchanges.
"""
import numpy as np
import pytest

import harness
from opensbli_gb300 import abi, problems

pytestmark = pytest.mark.gpu

BCS = {"zero_grad": (abi.BC_ZERO_GRAD, abi.BC_ZERO_GRAD), "extrap": (abi.BC_EXTRAP1, abi.BC_EXTRAP0),
       "periodic": (abi.BC_PERIODIC, abi.BC_PERIODIC)}


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 1e-5)])
@pytest.mark.parametrize("depth", [[1, 2], [2, 2], [3, 1], [3, 3]])
@pytest.mark.parametrize("bc", sorted(BCS))
@pytest.mark.parametrize("n", [30, 400])
def test_depth_below_the_stencil(built_lib, oracle_lib, n, bc, depth, precision, tol):
    from opensbli_gb300.solver import Solver
    spec, q = problems.sod(n, scheme=abi.SCHEME_WENO5_JS, bc=BCS[bc])
    spec.bc_depth = [depth]
    rng = np.random.default_rng(9)
    q = [a * (1.0 + 5e-2 * rng.uniform(-1.0, 1.0, a.shape)) for a in q]
    q[1] += 0.05 * rng.uniform(-1.0, 1.0, q[1].shape)
    dt = 0.05 / n
    s = Solver([(spec, q)], precision=precision, rk="ls3")
    s.step(dt, 3)
    got = s.state(0)
    s.close()
    ob = harness.OracleBlocks([(spec, q)])
    ob.apply_bc()
    ob.step(abi.RK_LOW_STORAGE, problems.RK3_LS_A, problems.RK3_LS_B, dt, 3)
    for v in range(3):
        assert harness.rel_err(got[v], ob.q[0][v]) < tol, v
