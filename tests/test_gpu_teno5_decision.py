"""TENO5's cut-off decision in FP64 3D blocks on windows whose outer indicators agree to 1e-7 while
the third is smaller still: a front that runs out into nearly flat gas.  Their difference is then far
above FP64's rounding but only the rounding of an FP32 evaluation, so the decision must not be taken
in FP32 (teno5_mask).

A contact (uniform velocity and pressure) carries such windows in the density along one axis, random
ones in every row.  The windows: differences d1 = 2 d2 (1 + t), d3 ~ 0 and d4, with tau / b0 = 2.5 t
between 6e-8 and 2.5e-7 and tau / b1 between 10.5 and 30, where the outer stencils go (the cut-off of
1e-6 lies at 9): a decision to keep them moves the flux by 0.05 d2.  Tolerance 1e-12 of the largest
residual, as for the other FP64 residuals: rounding moves tau by 1e-7 of itself at most, so no decision
depends on it.
"""
import numpy as np
import pytest

import harness
from opensbli_gb300 import abi, problems
from opensbli_gb300.spec import BlockSpec

pytestmark = pytest.mark.gpu

PERIOD = 16


def near_tie_contact(axis, sign):
    size = [8, 8, 8]
    size[axis] = 8 * PERIOD
    spec = BlockSpec(ndim=3, size=tuple(size), scheme=abi.SCHEME_TENO5, averaging=abi.AVG_ROE,
                     delta=tuple(1.0 / n for n in size), gama=1.4, eps=1e-40)
    rng = np.random.default_rng(7)
    shape = (8, 8, 8)  # rows of the two other axes, windows of a row
    d2 = 0.05 * rng.uniform(0.3, 1.0, shape) * rng.choice([-1.0, 1.0], shape)
    tau = 10.0 ** rng.uniform(np.log10(6e-8), np.log10(2.5e-7), shape)  # over b0 = 4/3 d2^2
    ratio = rng.uniform(10.5, 30.0, shape)
    d = [2.0 * d2 * (1.0 + 0.4 * tau), d2, 1e-9 * d2, d2 * np.sqrt(tau / ratio)]  # b0 = 4/3 d2^2, b1 = 4/3 d4^2
    steps = np.zeros(shape + (PERIOD,))
    for k in range(4):
        steps[..., 4 + k] = d[k]
    back = rng.uniform(0.5, 1.5, shape + (PERIOD - 4,))  # the way back in uneven steps
    back *= -(sum(d) / back.sum(-1))[..., None]
    steps[..., :4], steps[..., 8:] = back[..., :4], back[..., 4:]
    rho = 1.0 + np.cumsum(steps.reshape(8, 8, -1), -1)
    if sign < 0:
        rho = rho[..., ::-1]
    rho = np.moveaxis(rho, -1, 2 - axis)  # arrays are z, y, x
    full = np.ones(spec.shape)
    full[spec.interior()] = rho
    one = np.ones(spec.shape)
    return spec, problems._cons(spec, full, [(sign * 0.5 if i == axis else 0.0) * one for i in range(3)], one)


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("sign", [1, -1])
def test_near_ties_fp64(built_lib, oracle_lib, axis, sign):
    from opensbli_gb300.solver import Solver
    spec, q = near_tie_contact(axis, sign)
    s = Solver([(spec, q)], precision="fp64")
    s.apply_bc()
    got = s.residual(0)
    s.close()
    ob = harness.OracleBlocks([(spec, q)])
    ob.apply_bc()
    ref = ob.residual(0)
    sl = spec.interior()
    scale = max(float(np.max(np.abs(r[sl]))) for r in ref)
    for v in range(5):
        assert float(np.max(np.abs(got[v][sl] - ref[v][sl]))) < 1e-12 * scale, v
