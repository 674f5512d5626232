"""How the resident 1D path shares blocks out among CTAs, at the ends of its rules: as many blocks as
SMs with the largest one it takes (the clusters shrink to as few CTAs as hold the block).  Against the
per-block path in the same precision, tolerances as in test_gpu_resident.py: FP64 1e-13 (the same
operations on the same values, contracted differently at most), FP32 1e-5."""
import numpy as np
import pytest

import harness
from opensbli_gb300 import abi, problems

pytestmark = pytest.mark.gpu


def _advance(blocks, precision, dt, mode=None):
    from opensbli_gb300.solver import Solver
    s = Solver(blocks, precision=precision, rk="ls3")
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


def _tubes(sizes):
    rng = np.random.default_rng(4)
    blocks = []
    for n in sizes:
        spec, q = problems.sod(n, scheme=abi.SCHEME_WENO5_Z)
        blocks.append((spec, [a * (1.0 + 1e-2 * rng.standard_normal(a.shape)) for a in q]))
    return blocks


def _check(blocks):
    dt = 0.05 / max(spec.size[0] for spec, _ in blocks)
    for precision, tol in (("fp64", 1e-13), ("fp32", 1e-5)):
        per, _ = _advance(blocks, precision, dt, abi.SCHED_PER_BLOCK)
        got, launches = _advance(blocks, precision, dt)
        assert launches == 1
        for i, (spec, _) in enumerate(blocks):
            for v in range(spec.nvars):
                assert harness.rel_err(got[i][v], per[i][v]) < tol, (precision, i, v)


@pytest.mark.parametrize("largest", [2990, 2897, 2896])
def test_as_many_blocks_as_sms(built_lib, largest):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    _check(_tubes([6] * (sms - 1) + [largest]))
