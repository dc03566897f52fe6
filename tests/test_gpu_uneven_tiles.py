"""Tiles whose particles do not lie evenly over their cells: crowded cells, layers
one cell thick, bodies that end in a tile.

One step against the oracle around the counts where a warp's run changes (whole
chunks of 16 and 32 particles for each of 4, 8 or 16 warps): 1e-10 of each field's
scale plus 100x the oracle's own spread under a few-ulp perturbation, as the other
one-step parity tests.  And times against a scene of the same particles that fill
their tiles evenly: the same sums, so the factor allows for the flushes of shared
patches, not for warps that idle."""
import numpy as np
import pytest

from matter_tests_b200 import scenes
from matter_tests_b200.abi import BC, PREC_FP64, PREC_MIXED
from matter_tests_b200.gpu import GpuSim

import cases
from gpu_util import compare_states, needs_gpu, oracle_sensitivity, run_gpu, run_oracle

pytestmark = [pytest.mark.gpu, needs_gpu]


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("musl", [0, 1])
@pytest.mark.parametrize("n", [63, 64, 65, 127, 129, 255, 256, 257, 511, 513, 700])
def test_one_crowded_cell(dim, musl, n):
    sc = cases.apply(cases.block(dim, 3, n=10 if dim == 3 else 20), use_musl=musl, flip_ratio=-0.95, **cases.MODEL_CASES["dp"])
    rng = np.random.default_rng(n)
    cells = np.full((n, dim), 5.0)
    cells[::9] = rng.integers(3, 9, size=cells[::9].shape)  # some in the cells around it
    sc.x = np.ascontiguousarray((cells + rng.uniform(0.05, 0.95, size=cells.shape)) * sc.params.dx)
    for k in ("v", "F", "B", "scalars"):
        setattr(sc, k, np.ascontiguousarray(getattr(sc, k)[:n]))
    sc = cases.box_plates(sc, BC.SlipFree, 0.3)
    g, o = run_gpu(sc, 1), run_oracle(sc, 1)
    compare_states(g, o, 1e-10, sens=oracle_sensitivity(sc, 1))


def _step_ms(x, prec):
    """Least time of the two scatters of a MUSL step."""
    sc = cases.apply(cases.block(3, 3, n=4), use_musl=1, precision=prec, **cases.MODEL_CASES["dp"])
    g = GpuSim(sc.params)
    g.upload(x)
    g.set_objects([], [])
    g.step(2)
    ms = []
    for _ in range(5):
        t = dict(g.profile(1))
        ms.append(t["k_p2g"] + t["k_g2p_musl"])
    g.close()
    return min(ms)


def _lattice(cells):
    return scenes.lattice([0.0] * 3, [0.01 * c for c in cells], 0.01, 2, np.random.default_rng(1))


@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED])
def test_layer_in_x_costs_as_a_layer_in_z(prec):
    assert _step_ms(_lattice([1, 400, 300]), prec) <= 1.4 * _step_ms(_lattice([400, 300, 1]), prec)


@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED])
def test_one_crowded_cell_in_a_large_scene(prec):
    x = _lattice([50, 50, 50])
    crowd = 0.07 + np.random.default_rng(2).uniform(0.0002, 0.0098, size=(3000, 3))
    assert _step_ms(np.concatenate([x, crowd]), prec) <= 1.6 * _step_ms(x, prec)


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("deg", [2, 3])
@pytest.mark.parametrize("n", [63, 65, 129, 257, 513, 700])
def test_transfer_sums_in_the_mixed_form(dim, deg, n):
    """Node mass and momentum of an uneven tile against the oracle.  A node sums at
    most n products of about 8 roundings of 6e-8 each, of any sign: 1e-5 of the
    largest is over 6 standard errors at n = 700."""
    sc = cases.apply(cases.block(dim, deg, n=10 if dim == 3 else 20), precision=PREC_MIXED, gravity=(0.0, 0.0, 0.0),
                     plastic_model=cases.PM.NoPlasticity)
    rng = np.random.default_rng(n)
    cells = np.full((n, dim), 5.0)
    cells[::9] = rng.integers(3, 9, size=cells[::9].shape)
    sc.x = np.ascontiguousarray((cells + rng.uniform(0.05, 0.95, size=cells.shape)) * sc.params.dx)
    for k in ("v", "B", "scalars"):
        setattr(sc, k, np.ascontiguousarray(getattr(sc, k)[:n]))
    sc.F = None  # no stress: the grid velocity is the transferred one
    sc.plates, sc.objects = [], []
    g, o = run_gpu(sc, 1)["g"], run_oracle(sc, 1)["g"]
    assert np.abs(g["mass"] - o["mass"]).max() <= 1e-5 * o["mass"].max()
    p, q = g["mass"][:, None] * g["v"], o["mass"][:, None] * o["v"]
    assert np.abs(p - q).max() <= 1e-5 * np.abs(q).max()
