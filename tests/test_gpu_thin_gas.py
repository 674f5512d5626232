"""FP32 reconstruction in a gas of very small density: the absolute epsilons of the weights stand in the
units of waves divided by the density, whatever units a kernel reconstructs in.  A shear with jumps of
+-J = 0.03 under uniform density and pressure, against the C oracle.

The tangential momentum is checked, which the vorticity waves carry.  (The jumps reach the entropy wave
as J^2, whose epsilon is in units of the density, and come back through the mass flux as J^3.)  Tolerance
2e-4 of its largest residual: J^2 / 30 = 3e-5 from that path and 6e-8 / J times the reconstruction's
conditioning (about 10) from rounding; weights that took the jump's stencils as smooth move the flux by
a sixtieth of the jump.
"""
import numpy as np
import pytest

import harness
from opensbli_gb300 import abi, problems
from opensbli_gb300.spec import BlockSpec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("density", [1.0, 1e-8, 1e-14])
@pytest.mark.parametrize("ndim,axis", [(2, 0), (2, 1), (3, 0), (3, 1), (3, 2)])
@pytest.mark.parametrize("scheme", [abi.SCHEME_WENO5_JS, abi.SCHEME_WENO5_Z, abi.SCHEME_TENO5])
def test_shear_fp32(built_lib, oracle_lib, ndim, axis, scheme, density):
    from opensbli_gb300.solver import Solver
    size = (24, 20, 16)[:ndim]
    spec = BlockSpec(ndim=ndim, size=size, scheme=scheme, averaging=abi.AVG_ROE, delta=tuple(1.0 / n for n in size),
                     gama=1.4, eps=1e-40)
    one = np.ones(spec.shape)
    band = np.abs(2 * (spec.grid_index(axis) % size[axis]) + 1 - size[axis]) < size[axis] // 2
    u = [0.3 * one if i == axis else np.where(band, -0.03, 0.03) * one for i in range(ndim)]
    q = problems._cons(spec, density * one, u, density * one)
    s = Solver([(spec, q)], precision="fp32")
    s.apply_bc()
    got = s.residual(0)
    s.close()
    ob = harness.OracleBlocks([(spec, q)])
    ob.apply_bc()
    ref = ob.residual(0)
    sl = spec.interior()
    for i in range(ndim):
        if i != axis:
            scale = float(np.max(np.abs(ref[1 + i][sl])))
            assert float(np.max(np.abs(got[1 + i][sl] - ref[1 + i][sl]))) < 2e-4 * scale, i
