"""Large cells in scenes of many more particles than a window of their ordering
holds (65536 indices): members spread over all windows, in two far apart, and
close together.  Permutation bit-exact against a stable argsort; and a large cell
of a large scene is ordered in a time that does not grow with the scene."""
import numpy as np
import pytest

from matter_tests_b200 import scenes
from matter_tests_b200.gpu import GpuSim

import cases
from gpu_util import needs_gpu

pytestmark = [pytest.mark.gpu, needs_gpu]

WINDOW = 65536


def _scene(dim, side, members, where, seed=2):
    """A lattice of 2^dim particles a cell and `members` more in one of its cells, at the indices `where` chooses."""
    sc = cases.apply(cases.block(dim, 2, n=4), plastic_model=cases.PM.NoPlasticity)
    dx, rng = sc.params.dx, np.random.default_rng(seed)
    x = scenes.lattice([0.0] * dim, [side * dx] * dim, dx, 2, rng)
    crowd = (3.0 + rng.uniform(0.1, 0.9, size=(members, dim))) * dx
    n = len(x) + members
    at = {"spread": lambda: rng.choice(n, members, replace=False),
          "ends": lambda: np.concatenate([np.arange(members // 2), n - 1 - np.arange(members - members // 2)]),
          "edge": lambda: WINDOW - members // 2 + np.arange(members),
          "together": lambda: n // 2 + np.arange(members)}[where]()
    out = np.empty((n, dim))
    mask = np.zeros(n, dtype=bool)
    mask[at] = True
    out[mask], out[~mask] = rng.permutation(crowd), rng.permutation(x) if where == "spread" else x
    sc.x = out
    sc.v = sc.F = sc.B = sc.scalars = None
    return sc


def _sim(sc):
    g = GpuSim(sc.params)
    g.upload(sc.x)
    g.set_objects([], [])
    return g


@pytest.mark.parametrize("dim,side", [(2, 200), (3, 28)])
@pytest.mark.parametrize("where", ["spread", "ends", "edge", "together"])
@pytest.mark.parametrize("members", [1025, 5000])
def test_members_over_windows_bitexact(dim, side, where, members):
    sc = _scene(dim, side, members, where)
    assert sc.Np > 2 * WINDOW
    g = _sim(sc)
    for _ in range(2):  # as uploaded, and in the order that the first step leaves
        g.step(1)
        keys, perm, ids = g.sort_state()
        np.testing.assert_array_equal(perm, np.argsort(keys, kind="stable"))
    g.close()


def test_time_does_not_grow_with_the_scene():
    """Ordering 3000 members takes three passes over them; it stays within 10 times the kernel's time without them."""
    ms = []
    for members in (0, 3000):
        g = _sim(_scene(3, 50, members, "spread"))
        g.step(2)
        ms.append(min(dict(g.profile(1))["k_sort_rank"] for _ in range(5)))
        g.close()
    assert ms[1] <= 10.0 * ms[0], ms
