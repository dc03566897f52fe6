"""The counting sort of cell keys: keys and stable permutation bit-exact against
the oracle's keys and a stable argsort, where its cells are small, at the size
from which a whole block orders a cell, and beyond; batched too."""
import numpy as np
import pytest

import cases
from gpu_util import needs_gpu, run_gpu, run_oracle

pytestmark = [pytest.mark.gpu, needs_gpu]

BIG = 1024  # largest cell ranked particle by particle


def _crowded(dim, counts, seed=1):
    """A block with counts[i] more particles in the middle of its i-th cells, in shuffled input order."""
    sc = cases.apply(cases.block(dim, 2, n=5 if dim == 3 else 9, seed=seed), plastic_model=cases.PM.DP, M=0.6)
    rng = np.random.default_rng(seed)
    dx = sc.params.dx
    add = []
    for i, c in enumerate(counts):
        corner = np.zeros(dim)
        corner[i % dim] = (i // dim + 1) * dx
        add.append(corner + dx * rng.uniform(0.3, 0.7, size=(c, dim)))
    x = np.concatenate([sc.x] + add)
    order = rng.permutation(len(x))
    sc.x = np.ascontiguousarray(x[order])
    sc.v, sc.F, sc.B, sc.scalars = None, None, None, None
    return sc


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("counts", [[], [1], [BIG - 40, BIG + 1], [3000, BIG, 1500, 1100]])
def test_sort_of_crowded_cells_bitexact(dim, counts):
    sc = _crowded(dim, counts)
    g, o = run_gpu(sc, 1), run_oracle(sc, 1)
    keys, perm, ids = g["sort"]
    np.testing.assert_array_equal(ids, np.arange(sc.Np))
    np.testing.assert_array_equal(keys, o["keys"])
    np.testing.assert_array_equal(perm, np.argsort(o["keys"], kind="stable"))


def test_sort_of_crowded_cells_in_a_batch():
    from matter_tests_b200.gpu import GpuBatch, GpuSim
    scs = [_crowded(3, [2000, 1100]), _crowded(3, []), _crowded(2, [1025])]
    sims = []
    for sc in scs:
        g = GpuSim(sc.params)
        g.upload(sc.x)
        g.set_scene_objects(sc)
        sims.append(g)
    batch = GpuBatch(sims)
    batch.step(1)
    for sc, g in zip(scs, sims):
        keys, perm, _ = g.sort_state()
        np.testing.assert_array_equal(perm, np.argsort(keys, kind="stable"))
    batch.close()
    for g in sims:
        g.close()
