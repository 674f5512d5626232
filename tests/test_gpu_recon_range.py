"""FP64 reconstructions over the range of values: the TENO5 decision taken in FP32 with its FP64
fallback, and the WENO common denominator with its wide-range form, against the C oracle.

The units move the values across the lines between those forms (differences from 1e-12 to 1e25);
half of every block is exactly uniform, so stencils with vanishing indicators sit next to a jump and
to a perturbed region.  Tolerance 1e-12 of the largest value per variable, as for the other FP64
parity tests: both sides round a stage's flux differences to about 1e-15 of the flux, and the
stage moves the state by less than its own size.
"""
import numpy as np
import pytest

import harness
from opensbli_gb300 import abi, problems
from opensbli_gb300.spec import BlockSpec

pytestmark = pytest.mark.gpu

SCHEMES = {"weno5js": abi.SCHEME_WENO5_JS, "weno5z": abi.SCHEME_WENO5_Z, "teno5": abi.SCHEME_TENO5}


@pytest.mark.parametrize("speed", [1.0, 1e-6, 340.0, 1e5, 1e12])
@pytest.mark.parametrize("ndim,avg", [(1, abi.AVG_SIMPLE), (2, abi.AVG_ROE), (3, abi.AVG_ROE), (3, abi.AVG_SIMPLE)])
@pytest.mark.parametrize("scheme", list(SCHEMES))
def test_recon_fp64_over_the_range(built_lib, oracle_lib, scheme, ndim, avg, speed):
    from opensbli_gb300.solver import Solver
    size = {1: (61,), 2: (37, 22), 3: (19, 13, 11)}[ndim]
    spec = BlockSpec(ndim=ndim, size=size, scheme=SCHEMES[scheme], averaging=avg, delta=tuple(1.0 / n for n in size),
                     gama=1.4)
    rng = np.random.default_rng(5)
    x = spec.grid_index(0) / size[0] + np.zeros(spec.shape)
    half = x < 0.5
    noise = [np.where(half, 0.0, 1e-2 * rng.standard_normal(spec.shape)) for _ in range(ndim + 2)]
    rho = np.where(half, 1.0, 0.4) * (1.0 + noise[0])
    u = [speed * ((0.3, -0.2, 0.1)[i] + noise[1 + i]) for i in range(ndim)]
    p = speed * speed * np.where(half, 1.0, 0.25) * (1.0 + noise[-1])
    q = problems._cons(spec, rho, u, p)
    dt = 0.02 / (max(size) * speed)
    s = Solver([(spec, q)], precision="fp64", rk="ls3")
    s.step(dt, 1)
    got = s.state(0)
    s.close()
    ob = harness.OracleBlocks([(spec, q)])
    ob.apply_bc()
    ob.step(abi.RK_LOW_STORAGE, problems.RK3_LS_A, problems.RK3_LS_B, dt, 1)
    sl = spec.interior()
    for v in range(spec.nvars):
        scale = max(float(np.max(np.abs(ob.q[0][w][sl]))) for w in (range(1, ndim + 1) if 1 <= v <= ndim else [v]))
        err = float(np.max(np.abs(got[v][sl] - ob.q[0][v][sl]))) / scale
        assert err < 1e-12, (v, err)
