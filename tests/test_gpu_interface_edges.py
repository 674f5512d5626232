"""Halos where two interface faces of a block meet: one value whatever the threads' order, the one
that the C oracle leaves.  The four-block layout has such edges on its first block.

osb_apply_bc only copies, so random states (halos included) have to agree with the oracle exactly,
and two runs of osb_step with each other."""
import numpy as np
import pytest

import harness
from opensbli_gb300 import problems

pytestmark = pytest.mark.gpu

SIZES = {"A": (16, 12, 8), "B": (12, 12, 8), "C": (16, 10, 8), "D": (14, 12, 8)}


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("seed", [0, 1, 2])
def test_apply_bc(built_lib, oracle_lib, precision, seed):
    from opensbli_gb300.solver import Solver
    rng = np.random.default_rng(seed)
    blocks = [(spec, [rng.uniform(1.0, 2.0, a.shape) for a in q], met)
              for spec, q, met in problems.curvilinear_multiblock_3d(sizes=SIZES)]
    s = Solver(blocks, precision=precision)
    s.apply_bc()
    got = [s.state(i) for i in range(4)]
    s.close()
    ob = harness.OracleBlocks(blocks)
    ob.apply_bc()
    for i in range(4):
        for v in range(5):
            assert np.array_equal(got[i][v], ob.q[i][v]), (i, v)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_steps_repeat(built_lib, precision):
    from opensbli_gb300.solver import Solver
    blocks = problems.curvilinear_multiblock_3d(sizes={"A": (64, 48, 16), "B": (32, 48, 16), "C": (64, 32, 16),
                                                       "D": (32, 48, 16)}, seed=4)
    runs = []
    for _ in range(3):
        s = Solver(blocks, precision=precision, rk="ls3")
        s.step(2e-3, 3)
        runs.append([s.state(i) for i in range(4)])
        s.close()
    for r in runs[1:]:
        for a, b in zip(r, runs[0]):
            for v in range(5):
                assert np.array_equal(a[v], b[v]), v
