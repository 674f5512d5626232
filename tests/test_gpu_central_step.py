"""osb_step on periodic central-scheme blocks, which are read in place between the stages (k_central WRAP)
and cut into z chunks of any length: sizes at the edges of the 32 x 8 columns, against the C oracle.
After the call the halos are those that osb_apply_bc gives, and the reductions, which read them, agree.

Tolerances: FP64 1e-12 of the largest value (of the three momenta for each of them), as for the other
FP64 parity tests; FP32 1e-6 (fluxes of at most 10 rounded to 6e-8, dt / Delta below 2e-2, six stages,
with room for the stencils' weights).
"""
import numpy as np
import pytest

import harness
from opensbli_gb300 import abi, problems

pytestmark = pytest.mark.gpu

SIZES = [(33, 9, 7), (31, 17, 6), (64, 8, 13), (6, 6, 6), (97, 7, 12), (24, 24, 24), (12, 12, 40)]
DT = 1e-3


def _block(sizes, split, viscous):
    spec, q = problems.tgv(sizes=sizes, minf=0.5, scheme=abi.SCHEME_CENTRAL4, viscous=viscous)
    spec.split_form = split
    rng = np.random.default_rng(21)
    return spec, [a * (1.0 + 1e-2 * rng.standard_normal(a.shape)) for a in q]


def _oracle(spec, q):
    ob = harness.OracleBlocks([(spec, q)])
    ob.apply_bc()
    ob.step(abi.RK_LOW_STORAGE, problems.RK3_LS_A, problems.RK3_LS_B, DT, 2)
    ob.apply_bc()
    return ob


def _check(spec, got, ref, tol):
    sl = spec.interior()
    for v in range(5):
        scale = max(float(np.max(np.abs(ref[w][sl]))) for w in ((1, 2, 3) if 1 <= v <= 3 else (v,)))
        assert float(np.max(np.abs(got[v][sl] - ref[v][sl]))) < tol * scale, v


@pytest.mark.parametrize("sizes", SIZES)
@pytest.mark.parametrize("split,viscous", [(abi.SPLIT_FEIEREISEN, abi.VISC_CONSTANT), (abi.SPLIT_FEIEREISEN, abi.VISC_NONE),
                                           (abi.SPLIT_KGP, abi.VISC_SUTHERLAND), (abi.SPLIT_KGP, abi.VISC_CONSTANT)])
@pytest.mark.parametrize("graphs", [True, False])
def test_step_fp64(built_lib, oracle_lib, sizes, split, viscous, graphs):
    from opensbli_gb300.solver import Solver
    spec, q = _block(sizes, split, viscous)
    s = Solver([(spec, q)], precision="fp64", rk="ls3", graphs=graphs)
    s.step(DT, 2)
    got = s.state(0)
    reds = {w: s.reduce(w) for w in (abi.RED_KE, abi.RED_ENSTROPHY_DISS, abi.RED_DILATATION_DISS)}
    s.apply_bc()
    again = s.state(0)
    s.close()
    ob = _oracle(spec, q)
    _check(spec, got, ob.q[0], 1e-12)
    for v in range(5):
        assert np.array_equal(got[v], again[v]), v
    for w, r in reds.items():
        assert abs(r - ob.reduce(w)) < 1e-12 * abs(ob.reduce(w)), w


@pytest.mark.parametrize("sizes", SIZES)
@pytest.mark.parametrize("split,viscous", [(abi.SPLIT_FEIEREISEN, abi.VISC_CONSTANT), (abi.SPLIT_KGP, abi.VISC_SUTHERLAND)])
@pytest.mark.parametrize("bulk", [0, 1])
def test_step_fp32(built_lib, oracle_lib, sizes, split, viscous, bulk):
    from opensbli_gb300.solver import Solver
    spec, q = _block(sizes, split, viscous)
    s = Solver([(spec, q)], precision="fp32", rk="ls3")
    s.set_central_staging(bulk)
    s.step(DT, 2)
    got = s.state(0)
    s.apply_bc()
    again = s.state(0)
    s.close()
    _check(spec, got, _oracle(spec, q).q[0], 1e-6)
    for v in range(5):
        assert np.array_equal(got[v], again[v]), v
