"""The scatters and gathers where their shortcuts end: particles on grid lines
(weights of exactly zero), a hair inside a cell's corner (weights under the
1e-25 threshold that mass and momentum skip), particle counts around the sizes
of a unit, a warp and a block, and crowded next to empty cells.

One step against the oracle, particles and grid: 1e-10 of each field's scale
plus 100x the oracle's own spread under a few-ulp perturbation, as the other
one-step parity tests."""
import numpy as np
import pytest

from matter_tests_b200.abi import BC

import cases
from gpu_util import compare_states, needs_gpu, oracle_sensitivity, run_gpu, run_oracle

pytestmark = [pytest.mark.gpu, needs_gpu]


def _place(sc, x, seed=3):
    """The scene's particles moved to x (its first len(x) particles)."""
    n = len(x)
    sc.x = np.ascontiguousarray(x)
    for k in ("v", "F", "B", "scalars"):
        setattr(sc, k, np.ascontiguousarray(getattr(sc, k)[:n]))
    return sc


def _block(dim, deg, musl, model="dp", n=None):
    sc = cases.apply(cases.block(dim, deg, n=n or (6 if dim == 3 else 12)), use_musl=musl, flip_ratio=-0.95,
                     **cases.MODEL_CASES[model])
    return cases.box_plates(sc, BC.SlipFree, 0.3)


def _check(sc):
    g, o = run_gpu(sc, 1), run_oracle(sc, 1)
    compare_states(g, o, 1e-10, sens=oracle_sensitivity(sc, 1))


@pytest.mark.parametrize("dim,deg", [(2, 2), (2, 3), (3, 2), (3, 3)])
@pytest.mark.parametrize("musl", [0, 1])
@pytest.mark.parametrize("model", ["dp", "dpvisc_mibf"])
@pytest.mark.parametrize("offset", [0.0, 1e-9, 1e-4, 0.5])
def test_particles_on_and_beside_grid_lines(dim, deg, musl, model, offset):
    sc = _block(dim, deg, musl, model)
    dx = sc.params.dx
    rng = np.random.default_rng(17)
    cells = rng.integers(0, 6, size=sc.x.shape)
    x = cells * dx + offset * dx * rng.choice([-1.0, 1.0], size=cells.shape)
    x[0] = 0.0  # the grid's origin is two cells left of the least coordinate
    _check(_place(sc, np.maximum(x, 0.0)))


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("musl", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 33, 64, 129, 257])
def test_particle_counts_around_the_shapes(dim, musl, n):
    sc = _block(dim, 3, musl, n=9 if dim == 3 else 14)
    rng = np.random.default_rng(n)
    _check(_place(sc, rng.uniform(0.0, 2.0, size=(n, dim)) * sc.params.dx))


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("musl", [0, 1])
def test_crowded_cells_between_empty_ones(dim, musl):
    sc = _block(dim, 2, musl, n=8 if dim == 3 else 20)
    rng = np.random.default_rng(2)
    n = min(sc.Np, 900)
    cells = np.where(rng.uniform(size=(n, 1)) < 0.8, 5, rng.integers(0, 5, size=(n, dim)) * 3)
    _check(_place(sc, (cells + rng.uniform(0.01, 0.99, size=(n, dim))) * sc.params.dx))


@pytest.mark.parametrize("threads", [32, 64, 96, 256])
def test_block_sizes_of_the_scatters(threads):
    from matter_tests_b200.gpu import GpuSim
    sc = _block(3, 3, 1, "dpmui")
    o = run_oracle(sc, 1)
    g = GpuSim(sc.params)
    g.upload(sc.x, sc.v, sc.F, sc.B, sc.scalars)
    g.set_scene_objects(sc)
    g.tile_threads = {"p2g": threads, "musl": min(threads, 128)}
    g.keep_pic_flip(True)
    g.step(1)
    out = dict(p=g.particles(pic_flip=True), g=g.grid(), c=g.clock())
    g.close()
    compare_states(out, o, 1e-10, sens=oracle_sensitivity(sc, 1))
