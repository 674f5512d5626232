"""The resident 1D path (one launch per osb_step call for small 1D blocks, state in shared
memory) against the per-block path and the oracle: every boundary kind, both RK schemes, and a
batch of independent blocks of different sizes."""
import numpy as np
import pytest

import harness
from opensbli_gb300 import abi, problems

pytestmark = pytest.mark.gpu

BCS = {"zero_grad": (abi.BC_ZERO_GRAD, abi.BC_ZERO_GRAD), "extrap": (abi.BC_EXTRAP1, abi.BC_EXTRAP0),
       "periodic": (abi.BC_PERIODIC, abi.BC_PERIODIC)}


def _run(blocks, rk, dt, steps, mode):
    from opensbli_gb300.solver import Solver
    s = Solver(blocks, precision="fp64", rk=rk)
    if mode is not None:
        s.set_schedule(mode=mode)
    s.apply_bc()
    n0 = s.launches()
    s.step(dt, steps)
    s.sync()
    out = [s.state(i) for i in range(len(blocks))]
    launches = s.launches() - n0
    s.close()
    return out, launches


@pytest.mark.parametrize("bc", sorted(BCS))
@pytest.mark.parametrize("rk", ["ls3", "sbli3"])
def test_resident_1d_matches_per_block_and_oracle(built_lib, oracle_lib, bc, rk):
    spec, q = problems.sod(150, bc=BCS[bc])
    dt, steps = 2e-4, 60
    res, nl = _run([(spec, q)], rk, dt, steps, None)
    assert nl == 1  # every stage of every step in one launch
    per, _ = _run([(spec, q)], rk, dt, steps, abi.SCHED_PER_BLOCK)
    kind, A, B = (abi.RK_LOW_STORAGE, problems.RK3_LS_A, problems.RK3_LS_B) if rk == "ls3" else \
        (abi.RK_SBLI3, problems.RK3_SBLI_NEW, problems.RK3_SBLI_OLD)
    ob = harness.OracleBlocks([(spec, q)])
    ob.apply_bc()
    ob.step(kind, A, B, dt, steps)
    sl = spec.interior()
    for v in range(spec.nvars):
        assert harness.rel_err(res[0][v][sl], ob.q[0][v][sl]) < 1e-12, (bc, rk, v)
        # halos too: the call leaves them as the per-block path does
        assert harness.rel_err(res[0][v], per[0][v]) < 1e-13, (bc, rk, v)


def test_resident_1d_batch_of_blocks(built_lib, oracle_lib):
    """Independent 1D blocks of different sizes, one CTA each, in the same launch."""
    blocks = [problems.sod(n) for n in (60, 400, 1000)]
    dt, steps = 1e-4, 40
    res, nl = _run(blocks, "ls3", dt, steps, None)
    assert nl == 1
    for i, (spec, q) in enumerate(blocks):
        ob = harness.OracleBlocks([(spec, q)])
        ob.apply_bc()
        ob.step(abi.RK_LOW_STORAGE, problems.RK3_LS_A, problems.RK3_LS_B, dt, steps)
        sl = spec.interior()
        errs = [harness.rel_err(res[i][v][sl], ob.q[0][v][sl]) for v in range(spec.nvars)]
        assert max(errs) < 1e-12, (i, errs)


@pytest.mark.parametrize("bc", ["zero_grad", "periodic"])
def test_resident_1d_fp32_residual(built_lib, oracle_lib, bc):
    """FP32-residual resident path: FP32 fluxes from an FP32 copy of the state, compensated
    flux differences, float-float dt x residual applied to the FP64 state.  Against the
    per-block FP32 path (the same arithmetic; 1e-5 of the field scale after 100 steps, as
    rounding differences near the shock move FP32 results by that much) and the FP64 oracle
    (the FP32-residual Sod tolerance, 1e-4).  The FP64 resident tests pin the logic at 1e-12."""
    spec, q = problems.sod(400, bc=BCS[bc])
    dt, steps = 2e-4, 100
    from opensbli_gb300.solver import Solver
    out = {}
    for mode in (None, abi.SCHED_PER_BLOCK):
        s = Solver([(spec, q)], precision="fp32", rk="ls3")
        if mode is not None:
            s.set_schedule(mode=mode)
        s.apply_bc()
        n0 = s.launches()
        s.step(dt, steps)
        s.sync()
        out[mode] = (s.state(0), s.launches() - n0)
        s.close()
    res, nl = out[None]
    per, _ = out[abi.SCHED_PER_BLOCK]
    assert nl == 1
    ob = harness.OracleBlocks([(spec, q)])
    ob.apply_bc()
    ob.step(abi.RK_LOW_STORAGE, problems.RK3_LS_A, problems.RK3_LS_B, dt, steps)
    sl = spec.interior()
    for v in range(spec.nvars):
        assert harness.rel_err(res[v][sl], per[v][sl]) < 1e-5, (bc, v, "per-block")
        assert harness.rel_err(res[v][sl], ob.q[0][v][sl]) < 1e-4, (bc, v, "oracle")


@pytest.mark.parametrize("bc", sorted(BCS))
@pytest.mark.parametrize("sizes", [(6,), (11, 12), (31,), (32, 33), (62, 63), (65, 6, 497), (511,), (2990, 6)])
def test_resident_1d_split_over_ctas(built_lib, oracle_lib, sizes, bc):
    """Sizes around the limits of the split of a block over the CTAs of a cluster (a warp of
    interfaces each, at least six points, blocks of very different sizes together), perturbed
    states: as the per-block path, halos included (1e-13: the same operations on the same values,
    contracted differently at most), and FP32 against FP64 within 1e-5 after two steps."""
    rng = np.random.default_rng(3)
    blocks = []
    for n in sizes:
        spec, q = problems.sod(n, scheme=abi.SCHEME_TENO5, bc=BCS[bc])
        blocks.append((spec, [a * (1.0 + 1e-2 * rng.standard_normal(a.shape)) for a in q]))
    dt = 0.05 / max(sizes)
    res, nl = _run(blocks, "ls3", dt, 2, None)
    assert nl == 1
    per, _ = _run(blocks, "ls3", dt, 2, abi.SCHED_PER_BLOCK)
    from opensbli_gb300.solver import Solver
    s = Solver(blocks, precision="fp32", rk="ls3")
    s.apply_bc()
    s.step(dt, 2)
    f32 = [s.state(i) for i in range(len(blocks))]
    s.close()
    for i, (spec, _) in enumerate(blocks):
        for v in range(spec.nvars):
            assert harness.rel_err(res[i][v], per[i][v]) < 1e-13, (i, v)
            assert harness.rel_err(f32[i][v], per[i][v]) < 1e-5, (i, v, "fp32")
