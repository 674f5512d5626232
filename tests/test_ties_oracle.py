"""teno5_ties.npz, states that a GPU computed, against the C oracle.

The shock tube has no tie that rounding decides: 1e-12 of the largest value, as between other FP64
paths.  In the shear layers the outer indicators of windows beside the layer tie, and each order of
operations, the oracle's included, keeps other stencils: 5e-3, as for the extruded layers.
"""
import os

import numpy as np
import pytest

import harness
from opensbli_gb300 import abi, problems
from opensbli_gb300.spec import BlockSpec

GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "teno5_ties.npz")


@pytest.mark.parametrize("name,size,tol", [("sod", (53,), 1e-12), ("kh", (24, 41), 5e-3), ("kh_fp32", (97, 60), 5e-3)])
def test_teno5_ties_against_oracle(oracle_lib, name, size, tol):
    g = np.load(GOLDEN)
    common = dict(ndim=len(size), size=size, scheme=abi.SCHEME_TENO5, gama=1.4, eps=1e-40)
    if name == "sod":
        z = abi.BC_ZERO_GRAD
        spec = BlockSpec(bc=[[z, z]], bc_depth=[[4, 4]], delta=[1.0 / 52], averaging=abi.AVG_SIMPLE, **common)
    else:
        spec = BlockSpec(delta=(1.0 / size[0], 1.0 / size[1]), averaging=abi.AVG_ROE, **common)
    ob = harness.OracleBlocks([(spec, list(g[name + "_q0"]))])
    ob.apply_bc()
    ob.step(abi.RK_LOW_STORAGE, problems.RK3_LS_A, problems.RK3_LS_B, float(g[name + "_dt"]), 9)
    sl = spec.interior()
    largest = max(float(np.max(np.abs(a[sl]))) for a in ob.q[0])
    for v in range(spec.nvars):
        assert float(np.max(np.abs(g[name + "_q"][v][sl] - ob.q[0][v][sl]))) < tol * largest, v
