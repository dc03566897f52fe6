"""Weights of 1e-25 and less carry no mass and no momentum (p2g.cpp:35, musl.cpp:51):
the nodes that only such a weight reaches stay exactly empty, where the small
weight is the third of a stencil clamped at the first node, and where it is a
subnormal FP32 number.

The empty nodes are the oracle's, exactly; the others agree within 1e-10 (FP64)
or 1e-5 (mixed) of the largest, as in the tests of the transfers."""
import itertools

import numpy as np
import pytest

from matter_tests_b200 import abi
from matter_tests_b200.abi import PREC_FP64, PREC_MIXED
from matter_tests_b200.gpu import load_library
from oracle.checkers import p2g_grid

import cases
from gpu_util import needs_gpu, run_gpu, run_oracle
from test_zz_no_alloc import _Call, _scene, _uniform_grid

pytestmark = [pytest.mark.gpu, needs_gpu]


def _corners(dim, values):
    return np.array(list(itertools.product(values, repeat=dim)))


@pytest.mark.parametrize("dim,deg", [(2, 2), (2, 3), (3, 2), (3, 3)])
@pytest.mark.parametrize("hair", [0.0, 1e-12, 1e-9, 1e-5])
def test_noalloc_beside_the_first_node(dim, deg, hair):
    """One particle a call: in the first cell of some axes, a hair past the first node, inside on the others."""
    p = _scene(dim, deg, n=4, seed=1).params
    dims = np.array((9, 10, 11)[:dim] + (1,) * (3 - dim))
    axes = _uniform_grid(dims, p.dx, (0.0, 0.0, 0.0))
    rng = np.random.default_rng(4)
    for u in _corners(dim, [hair, 2.3]):
        x = (u * p.dx)[None, :]
        v, B = rng.normal(size=(1, dim)), rng.normal(size=(1, dim * dim)) * p.dx
        om, ov, left = p2g_grid(p, x, v, B, *axes, dims)
        assert left == 0
        rc, m, vv, status = _Call(p, x, v, B, *axes, dims).run(load_library())
        assert rc == abi.MTR_OK and status == 0
        np.testing.assert_array_equal(m == 0.0, om == 0.0)
        assert np.all(vv[om == 0.0] == 0.0)
        assert np.abs(m - om).max() <= 1e-10 * om.max()
        assert np.abs(vv - ov).max() <= 1e-10 * np.abs(ov).max()


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("deg,hair", [(2, 1e-13), (3, 1e-13), (3, 1e-9)])
@pytest.mark.parametrize("musl", [0, 1])
@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED])
def test_step_beside_a_grid_line(dim, deg, hair, musl, prec):
    """Lone particles, 8 cells apart, a hair beside where a spline begins: a grid
    line (cubic) or the middle of a cell (quadratic)."""
    sc = cases.apply(cases.block(dim, deg, n=6 if dim == 3 else 12), use_musl=musl, flip_ratio=-0.95, precision=prec,
                     plastic_model=cases.PM.NoPlasticity, gravity=(0.0, 0.0, 0.0))
    line = 0.0 if deg == 3 else 0.5
    u = _corners(dim, [0.0, 8.0 + line + hair, 16.0 + line - hair, 24.0 + line + 0.3])
    sc.x = np.ascontiguousarray(u * sc.params.dx)
    for k in ("v", "B", "scalars"):
        setattr(sc, k, np.ascontiguousarray(getattr(sc, k)[:len(u)]))
    sc.F = None
    sc.plates, sc.objects = [], []
    g, o = run_gpu(sc, 1), run_oracle(sc, 1)
    rel = 1e-10 if prec == PREC_FP64 else 1e-5
    m, om = g["g"]["mass"], o["g"]["mass"]
    np.testing.assert_array_equal(m == 0.0, om == 0.0)
    assert np.abs(m - om).max() <= rel * om.max()
    assert np.all(g["g"]["v"][om == 0.0] == 0.0)
