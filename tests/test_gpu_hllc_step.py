"""osb_step with the HLLC-LM flux, whose sweeps do not carry the FP32 path's RK update: the state has to
advance all the same, on inviscid 2D and 3D blocks.

Against the C oracle: FP64 1e-12 of the largest value; FP32 2e-4 of the state's change, the tolerance of
FP32 residuals.
"""
import numpy as np
import pytest

import harness
from opensbli_gb300 import abi, problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("scheme", [abi.SCHEME_WENO5_JS, abi.SCHEME_WENO5_Z])
@pytest.mark.parametrize("ndim", [2, 3])
def test_hllc_advances(built_lib, oracle_lib, ndim, scheme, precision):
    from opensbli_gb300.solver import Solver
    if ndim == 2:
        spec, q = problems.kh(sizes=(33, 20), scheme=scheme)
    else:
        spec, q = problems.tgv(sizes=(18, 13, 11), minf=1.25, scheme=scheme, averaging=abi.AVG_ROE, viscous=abi.VISC_NONE)
    spec.flux_type = abi.FLUX_HLLC_LM
    rng = np.random.default_rng(8)
    q = [a * (1.0 + 1e-2 * rng.standard_normal(a.shape)) for a in q]
    dt = 0.1 * min(spec.delta)
    s = Solver([(spec, q)], precision=precision, rk="ls3")
    s.step(dt, 2)
    got = s.state(0)
    s.close()
    ob = harness.OracleBlocks([(spec, q)])
    ob.apply_bc()
    ob.step(abi.RK_LOW_STORAGE, problems.RK3_LS_A, problems.RK3_LS_B, dt, 2)
    sl = spec.interior()
    mom = range(1, 1 + ndim)
    for v in range(spec.nvars):
        group = mom if v in mom else (v,)
        if precision == "fp64":
            bound = 1e-12 * max(float(np.max(np.abs(ob.q[0][w][sl]))) for w in group)
        else:
            bound = 2e-4 * max(float(np.max(np.abs(ob.q[0][w][sl] - q[w][sl]))) for w in group)
        assert float(np.max(np.abs(got[v][sl] - ob.q[0][v][sl]))) < bound, v
