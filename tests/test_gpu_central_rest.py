"""Central schemes on gas at rest under uniform pressure with uneven density and temperature: the
energy is the same number at every point, so the pressure is too, its derivatives and with them the
momentum residual are exactly zero in any precision."""
import numpy as np
import pytest

from opensbli_gb300 import abi, problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("split", [abi.SPLIT_KGP, abi.SPLIT_FEIEREISEN])
@pytest.mark.parametrize("viscous", [abi.VISC_NONE, abi.VISC_CONSTANT, abi.VISC_SUTHERLAND])
def test_rest_under_uniform_pressure(built_lib, precision, split, viscous):
    from opensbli_gb300.solver import Solver
    spec, _ = problems.tgv(sizes=(33, 12, 9), minf=0.5, scheme=abi.SCHEME_CENTRAL4, viscous=viscous)
    spec.split_form = split
    rng = np.random.default_rng(6)
    zero = np.zeros(spec.shape)
    q = problems._cons(spec, rng.uniform(0.3, 3.0, spec.shape), [zero] * 3, 2.7 + zero)
    s = Solver([(spec, q)], precision=precision)
    s.apply_bc()
    got = s.residual(0)
    s.close()
    for v in (1, 2, 3):
        assert not np.any(got[v][spec.interior()]), v
