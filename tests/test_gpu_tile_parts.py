"""Scenes of few tiles have each tile's particles cut over 4 or 2 blocks, larger
ones have a block per tile: one step on both sides of the two particle counts
where the cut changes (148 and 296 tiles of 256 particles in 2D, of 512 in 3D).

Against the oracle: 1e-10 of each field's scale plus 100x the oracle's own
spread under a few-ulp perturbation, as the other one-step parity tests."""
import numpy as np
import pytest

from matter_tests_b200.abi import BC

import cases
from gpu_util import compare_states, needs_gpu, oracle_sensitivity, run_gpu, run_oracle

pytestmark = [pytest.mark.gpu, needs_gpu]


@pytest.mark.parametrize("dim,side,tile", [(2, 138, 256), (3, 27, 512)])
@pytest.mark.parametrize("musl", [0, 1])
@pytest.mark.parametrize("tiles", [148, 296])
@pytest.mark.parametrize("over", [0, 1])
def test_one_step_where_the_cut_changes(dim, side, tile, musl, tiles, over):
    sc = cases.apply(cases.block(dim, 2, n=side), use_musl=musl, flip_ratio=-0.95, **cases.MODEL_CASES["dp"])
    n = tiles * tile - 1 + over
    assert sc.Np >= n
    for k in ("x", "v", "F", "B", "scalars"):
        setattr(sc, k, np.ascontiguousarray(getattr(sc, k)[:n]))
    sc = cases.box_plates(sc, BC.SlipFree, 0.3)
    compare_states(run_gpu(sc, 1), run_oracle(sc, 1), 1e-10, sens=oracle_sensitivity(sc, 1))
