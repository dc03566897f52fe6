"""The grid coordinates (arange, tools.hpp:291-296) are a chain of rounded
additions; the step forms them 32 at a time.  Bit for bit against the oracle
over binades, through zero, with increments that are and are not
representable, from a few nodes to several thousand, and over steps in which
the grid moves and regrows."""
import numpy as np
import pytest

import cases
from gpu_util import needs_gpu, run_gpu, run_oracle

pytestmark = [pytest.mark.gpu, needs_gpu]


def _spread(lo, hi, dx, n=60, dim=2, v=0.0):
    sc = cases.apply(cases.block(dim, 2, n=4), plastic_model=cases.PM.NoPlasticity)
    rng = np.random.default_rng(5)
    p = sc.params
    p.dx = dx
    p.particle_volume = dx ** dim / 4
    p.particle_mass = 1000.0 * p.particle_volume
    x = rng.uniform(0.0, 3.0 * dx, size=(n, dim))
    x[:, 0] = np.linspace(lo, hi, n)
    sc.x = x
    sc.v = np.zeros((n, dim))
    sc.v[:, 0] = v * np.linspace(-1.0, 1.0, n)
    sc.F = sc.B = sc.scalars = None
    return sc


@pytest.mark.parametrize("lo,hi,dx", [
    (0.0, 1.0, 0.1), (0.0, 1.0, 0.0625), (-37.3, 41.7, 0.013), (-1e-3, 2.0, 0.001), (1e5, 1e5 + 20.0, 0.0371),
    (-0.3, 0.05, 1.0 / 3.0), (0.0, 0.7, 0.7 / 31.0), (0.0, 0.7, 0.7 / 32.0), (0.0, 0.7, 0.7 / 33.0)])
@pytest.mark.parametrize("steps", [1, 3])
def test_axes_bitwise(lo, hi, dx, steps):
    sc = _spread(lo, hi, dx)
    g, o = run_gpu(sc, steps), run_oracle(sc, steps)
    assert tuple(g["g"]["dims"]) == tuple(o["g"]["dims"])
    for k in ("x", "y"):
        assert np.array_equal(g["g"][k], o["g"][k]), k


def test_axes_bitwise_while_the_grid_grows():
    sc = _spread(0.0, 0.5, 0.011, v=40.0)
    for steps in (5, 17, 40):  # one graph and single steps
        g, o = run_gpu(sc, steps), run_oracle(sc, steps)
        assert g["c"]["step"] == o["c"]["step"] == steps
        assert tuple(g["g"]["dims"]) == tuple(o["g"]["dims"])
        for k in ("x", "y"):
            assert np.array_equal(g["g"][k], o["g"][k]), (k, steps)
