"""Cutting tiles over several blocks is for scenes that leave SMs idle.  A sparse
scene has few particles in many tiles: alone, where its tiles may be cut, its step
takes no longer than as the only member of a batch, whose tiles are not cut (the
margin is for the different launches of the two)."""
import time

import numpy as np
import pytest
import torch

from matter_tests_b200.abi import PREC_FP64, PREC_MIXED
from matter_tests_b200.gpu import GpuBatch, GpuSim

import cases
from gpu_util import needs_gpu

pytestmark = [pytest.mark.gpu, needs_gpu]


def _step_ms(advance):
    advance(16)
    ms = []
    for _ in range(5):
        torch.cuda.synchronize()
        t = time.perf_counter()
        advance(16)
        torch.cuda.synchronize()
        ms.append((time.perf_counter() - t) / 16 * 1e3)
    return min(ms)


@pytest.mark.parametrize("dim,side,n", [(2, 500, 5000), (3, 106, 20000), (3, 27, 20000)])
@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED])
def test_sparse_scene_alone_and_in_a_batch(dim, side, n, prec):
    sc = cases.apply(cases.block(dim, 3, n=4), use_musl=1, flip_ratio=-0.95, precision=prec, cfl_elastic=0.01, end_frame=1000,
                     **cases.MODEL_CASES["dp"])
    x = np.random.default_rng(1).uniform(0.0, side * sc.params.dx, size=(n, dim))
    ms = []
    for batched in (False, True):
        g = GpuSim(sc.params)
        g.upload(x)
        g.set_objects([], [])
        batch = GpuBatch([g]) if batched else None
        ms.append(_step_ms((batch or g).step))
        if batch:
            batch.close()
        g.close()
    assert ms[0] <= 1.15 * ms[1], ms
