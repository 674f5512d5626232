"""How the resident 1D path shares blocks out among CTAs, at the ends of its rules: as many blocks as
SMs with the largest one it takes (the clusters shrink to as few CTAs as hold the block), and FP32
blocks on either side of the line between one CTA and a cluster.  Against the per-block path in the
same precision, halos included (TENO5: WENO5-Z's outer indicators tie exactly at zero-gradient ends,
and two kernels' roundings then decide differently).  Tolerances as in test_gpu_resident.py: FP64 1e-13
(the same operations on the same values, contracted differently at most), FP32 1e-5."""
import numpy as np
import pytest

import harness
from opensbli_gb300 import abi, problems

pytestmark = pytest.mark.gpu


BCS = {"zero_grad": (abi.BC_ZERO_GRAD, abi.BC_ZERO_GRAD), "extrap": (abi.BC_EXTRAP1, abi.BC_EXTRAP0),
       "periodic": (abi.BC_PERIODIC, abi.BC_PERIODIC)}


def _advance(blocks, precision, dt, mode=None, rk="ls3"):
    from opensbli_gb300.solver import Solver
    s = Solver(blocks, precision=precision, rk=rk)
    if mode is not None:
        s.set_schedule(mode=mode)
    s.apply_bc()
    n0 = s.launches()
    s.step(dt, 2)
    s.sync()
    out = [s.state(i) for i in range(len(blocks))]
    launches = s.launches() - n0
    s.close()
    return out, launches


def _tubes(sizes, bc="zero_grad"):
    rng = np.random.default_rng(4)
    blocks = []
    for n in sizes:
        spec, q = problems.sod(n, scheme=abi.SCHEME_TENO5, bc=BCS[bc])
        blocks.append((spec, [a * (1.0 + 1e-2 * rng.standard_normal(a.shape)) for a in q]))
    return blocks


def _check(blocks, precisions=("fp64", "fp32"), rk="ls3"):
    dt = 0.05 / max(spec.size[0] for spec, _ in blocks)
    for precision in precisions:
        tol = 1e-13 if precision == "fp64" else 1e-5
        per, _ = _advance(blocks, precision, dt, abi.SCHED_PER_BLOCK, rk)
        got, launches = _advance(blocks, precision, dt, rk=rk)
        assert launches == 1
        for i, (spec, _) in enumerate(blocks):
            for v in range(spec.nvars):
                assert harness.rel_err(got[i][v], per[i][v]) < tol, (precision, i, v)


@pytest.mark.parametrize("largest", [2990, 2897, 2896])
def test_as_many_blocks_as_sms(built_lib, largest):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    _check(_tubes([6] * (sms - 1) + [largest]))


@pytest.mark.parametrize("bc", sorted(BCS))
@pytest.mark.parametrize("rk", ["ls3", "sbli3"])
@pytest.mark.parametrize("n", [6, 63, 244, 245])
def test_fp32_one_block(built_lib, n, rk, bc):
    _check(_tubes([n], bc), ("fp32",), rk)


@pytest.mark.parametrize("n,count", [(6, 305), (255, 76), (255, 75), (256, 76), (300, 256), (300, 220), (400, 150),
                                     (1000, 160), (1560, 256), (1610, 160)])
def test_fp32_many_blocks(built_lib, n, count):
    _check(_tubes([n] * count), ("fp32",))


def test_fp32_blocks_of_different_sizes(built_lib):
    _check(_tubes([1000] + [50] * 300), ("fp32",))
    _check(_tubes([244, 6, 63, 100]), ("fp32",))
