"""mtr_p2g_noalloc at particle counts around the sizes its scatter works in (16
staged particles, a warp, a block) and with cells crowded next to empty ones.

Node mass and momentum against the oracle's P2G, 1e-12 of the largest: a node
sums at most a few thousand products of about 20 roundings each, 2e-16 apiece."""
import numpy as np
import pytest

from matter_tests_b200 import abi
from matter_tests_b200.gpu import load_library
from oracle.checkers import p2g_grid

from gpu_util import needs_gpu
from test_zz_no_alloc import _Call, _scene, _uniform_grid

pytestmark = [pytest.mark.gpu, needs_gpu]


def _check(dim, deg, n, crowded, dims):
    p = _scene(dim, deg, n=4, seed=1).params
    rng = np.random.default_rng(n)
    dims = np.array(dims[:dim] + (1,) * (3 - dim))
    axes = _uniform_grid(dims, p.dx, (-0.3, 0.7, 0.1))
    cells = rng.integers(1, np.maximum(dims[:dim] - 3, 2), size=(n, dim))
    if crowded:
        cells = np.where(rng.uniform(size=(n, 1)) < 0.8, np.minimum(5, dims[:dim] - 3), 1 + (cells - 1) // 3 * 3)
    x = np.array([a[0] for a in axes[:dim]]) + (cells + rng.uniform(0.0, 1.0, size=(n, dim))) * p.dx
    v, B = rng.normal(size=(n, dim)), rng.normal(size=(n, dim * dim)) * p.dx
    om, ov, left = p2g_grid(p, x, v, B, *axes, dims)
    assert left == 0
    rc, m, vv, status = _Call(p, x, v, B, *axes, dims).run(load_library())
    assert rc == abi.MTR_OK and status == 0
    assert np.abs(m - om).max() <= 1e-12 * om.max()
    mom = om[:, None] * ov
    assert np.abs(m[:, None] * vv - mom).max() <= 1e-12 * np.abs(mom).max()


@pytest.mark.parametrize("dim,deg", [(2, 2), (2, 3), (3, 2), (3, 3)])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 33, 255, 257, 3000])
@pytest.mark.parametrize("crowded", [False, True])
def test_counts_and_crowding(dim, deg, n, crowded):
    _check(dim, deg, n, crowded, (13, 17, 11))


@pytest.mark.parametrize("dim,deg", [(2, 2), (3, 3)])
@pytest.mark.parametrize("over", [0, 1])
@pytest.mark.parametrize("crowded", [False, True])
def test_both_sides_of_the_tile_count_where_the_blocks_change(dim, deg, over, crowded):
    """148 and 149 tiles: a tile has four blocks of 256 threads, then two of 128."""
    tile = 4 if dim == 3 else 8
    dims = (149 * tile, tile, tile) if over else (74 * tile, 2 * tile, tile)
    _check(dim, deg, 5000, crowded, dims)
