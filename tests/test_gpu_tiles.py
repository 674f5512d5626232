"""Kernels at the edges of their tiles: the FP64 central kernel (32 x 8 columns, chunks of z), the
sweeps' line numbering and the reductions, on block sizes just below, at and above a tile, against
the C oracle.

Tolerances: FP64 1e-12 of the largest residual (sum) -- a few hundred roundings of 1.1e-16 of the
terms, which are of the residual's size on these perturbed fields times at most 1 / (k Delta) ~ 100.
FP32 residual 2e-4 of the largest residual: flux differences of FP32 fluxes, 2^-24 |F| / Delta against
residuals of the size of the perturbation's gradients (1e-2 |F| / Delta), times the reconstruction's
conditioning (about 10).
"""
import numpy as np
import pytest

import harness
from opensbli_gb300 import abi, problems

pytestmark = pytest.mark.gpu

SIZES = [(33, 9, 7), (31, 17, 6), (64, 8, 13), (32, 16, 20), (6, 6, 6), (97, 7, 12)]


def _block(sizes, scheme, viscous, seed, minf=0.5):
    spec, q = problems.tgv(sizes=sizes, minf=minf, scheme=scheme, averaging=abi.AVG_ROE, viscous=viscous)
    rng = np.random.default_rng(seed)
    q = [a * (1.0 + 1e-2 * rng.standard_normal(a.shape)) + (1e-2 * rng.standard_normal(a.shape) if 1 <= i <= 3 else 0.0)
         for i, a in enumerate(q)]
    return spec, q


def _residuals(spec, q, precision):
    from opensbli_gb300.solver import Solver
    ob = harness.OracleBlocks([(spec, q)])
    ob.apply_bc()
    s = Solver([(spec, q)], precision=precision)
    s.apply_bc()
    got = s.residual(0)
    red = {w: s.reduce(w) for w in (abi.RED_KE, abi.RED_ENSTROPHY_DISS, abi.RED_DILATATION_DISS, abi.RED_CFL_DT)}
    s.close()
    return got, ob.residual(0), red, {w: ob.reduce(w) for w in red}


@pytest.mark.parametrize("sizes", SIZES)
@pytest.mark.parametrize("conv,viscous", [("central", abi.VISC_CONSTANT), ("central", abi.VISC_SUTHERLAND),
                                          ("central", abi.VISC_NONE), ("teno5", abi.VISC_SUTHERLAND),
                                          ("teno5", abi.VISC_CONSTANT), ("teno5", abi.VISC_POWER_LAW)])
def test_central_fp64_tiles(built_lib, oracle_lib, sizes, conv, viscous):
    spec, q = _block(sizes, abi.SCHEME_CENTRAL4 if conv == "central" else abi.SCHEME_TENO5, viscous, 11)
    if viscous == abi.VISC_POWER_LAW:
        spec.visc_power, spec.forcing = 0.7, (-1.0, 0.25, 0.5)
    got, ref, red, ored = _residuals(spec, q, "fp64")
    sl = spec.interior()
    for v in range(5):
        scale = max(float(np.max(np.abs(ref[w][sl]))) for w in ((1, 2, 3) if 1 <= v <= 3 else (v,)))
        assert float(np.max(np.abs(got[v][sl] - ref[v][sl]))) < 1e-12 * scale, v
    for w in red:
        assert abs(red[w] - ored[w]) < 1e-12 * abs(ored[w]), w


@pytest.mark.parametrize("sizes", SIZES)
@pytest.mark.parametrize("scheme", [abi.SCHEME_WENO5_JS, abi.SCHEME_WENO5_Z, abi.SCHEME_TENO5])
def test_sweeps_fp32_lines(built_lib, oracle_lib, sizes, scheme):
    spec, q = _block(sizes, scheme, abi.VISC_NONE, 12, minf=1.25)
    got, ref, _, _ = _residuals(spec, q, "fp32")
    sl = spec.interior()
    for v in range(5):
        scale = max(float(np.max(np.abs(ref[w][sl]))) for w in ((1, 2, 3) if 1 <= v <= 3 else (v,)))
        d = np.abs(got[v][sl] - ref[v][sl])
        # TENO5's cut-off may flip where it is within FP32 rounding of its threshold: a few points
        bad = int(np.count_nonzero(d > 2e-4 * scale))
        assert bad <= (d.size // 500 if scheme == abi.SCHEME_TENO5 else 0), (v, bad, float(d.max()) / scale)


# k_flux_tile: 63 points of 8 rows along x, 15 points of 32 lines along y and z
@pytest.mark.parametrize("sizes", [(63, 8), (64, 9), (127, 33), (31, 16), (6, 7), (63, 8, 6), (33, 15, 16), (65, 7, 31)])
@pytest.mark.parametrize("scheme", [abi.SCHEME_WENO5_JS, abi.SCHEME_WENO5_Z, abi.SCHEME_TENO5, abi.SCHEME_TENO6])
@pytest.mark.parametrize("avg", [abi.AVG_ROE, abi.AVG_SIMPLE])
def test_sweeps_fp64_tiles(built_lib, oracle_lib, sizes, scheme, avg):
    if len(sizes) == 3:
        spec, q = _block(sizes, scheme, abi.VISC_NONE, 13, minf=1.25)
    else:
        spec, q = problems.kh(sizes=sizes, scheme=scheme)
        rng = np.random.default_rng(13)
        q = [a * (1.0 + 1e-2 * rng.standard_normal(a.shape)) for a in q]
    spec.averaging = avg
    got, ref, _, _ = _residuals(spec, q, "fp64")
    sl = spec.interior()
    mom = range(1, 1 + len(sizes))
    for v in range(spec.nvars):
        scale = max(float(np.max(np.abs(ref[w][sl]))) for w in (mom if v in mom else (v,)))
        assert float(np.max(np.abs(got[v][sl] - ref[v][sl]))) < 1e-12 * scale, v


# k_filter_flux lists the faces that are on among 512: none, some and all of them on; points selected
# whose faces are off.  Tolerance 1e-10 as the other filter tests (WENO3-Z with an epsilon of 1e-40).
@pytest.mark.parametrize("sizes", [(8, 8, 8), (7, 9, 11), (33, 16, 9)])
@pytest.mark.parametrize("check,select", [(0.05, 0.05), (0.0, 0.0), (0.3, 0.01), (0.01, 0.3), (2.0, 0.0)])
def test_filter_faces_fp64(built_lib, oracle_lib, sizes, check, select):
    from opensbli_gb300.solver import Solver
    spec, q = _block(sizes, abi.SCHEME_CENTRAL4, abi.VISC_SUTHERLAND, 14, minf=1.25)
    spec.split_form, spec.filter = abi.SPLIT_KGP, abi.FILTER_WENO3
    spec.ducros_check, spec.ducros_select = check, select
    s = Solver([(spec, q)], precision="fp64", rk="ls3")
    s.apply_bc()
    s.step(2e-3, 1)
    got = s.state(0)
    s.close()
    ob = harness.OracleBlocks([(spec, q)])
    ob.apply_bc()
    ob.step(abi.RK_LOW_STORAGE, problems.RK3_LS_A, problems.RK3_LS_B, 2e-3, 1)
    sl = spec.interior()
    errs = [harness.rel_err(got[v][sl], ob.q[0][v][sl]) for v in range(5)]
    assert max(errs) < 1e-10, errs
