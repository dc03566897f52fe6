"""A particle whose position is not finite, or lies far left of the grid, takes
no part in the transfers: the step reports MTR_STATUS_STENCIL_OOB and leaves the
grid and the other particles as if it were absent.

Both runs sum the same terms in another order: 1e-10 of each field's scale in
FP64 and 1e-5 in the mixed form, the tolerances of the batch tests."""
import numpy as np
import pytest

from matter_tests_b200.abi import BC, PREC_FP64, PREC_MIXED, STATUS_STENCIL_OOB

import cases
from gpu_util import needs_gpu, run_gpu

pytestmark = [pytest.mark.gpu, needs_gpu]

FIELDS = ("x", "v", "F", "B", "scalars")


def _lost_and_absent(sc, k, axis, value):
    """One step with particle k's coordinate replaced, and one without the particle."""
    sc.v[k] = 0.0
    keep = np.arange(sc.Np) != k
    full = {f: getattr(sc, f) for f in FIELDS}
    for f in FIELDS:
        setattr(sc, f, np.ascontiguousarray(full[f][keep]))
    want = run_gpu(sc, 1)
    for f in FIELDS:
        setattr(sc, f, full[f].copy())
    sc.x[k, axis] = value
    return run_gpu(sc, 1), want, keep


def _check(sc, k, axis, value):
    got, want, keep = _lost_and_absent(sc, k, axis, value)
    rel = 1e-10 if sc.params.precision == PREC_FP64 else 1e-5
    assert want["status"][0] == 0 and got["status"][0] == STATUS_STENCIL_OOB
    assert got["status"][1] == k
    assert tuple(got["g"]["dims"]) == tuple(want["g"]["dims"])
    pairs = [("grid " + f, got["g"][f], want["g"][f]) for f in ("mass", "v", "flip")]
    pairs += [(f, got["p"][f][keep], want["p"][f]) for f in ("x", "v", "F", "B")]
    for name, a, b in pairs:
        assert np.all(np.isfinite(a)), name
        assert np.abs(a - b).max() <= rel * np.abs(b).max(), name


@pytest.mark.parametrize("dim,axis", [(2, 0), (2, 1), (3, 0), (3, 1), (3, 2)])
@pytest.mark.parametrize("deg", [2, 3])
@pytest.mark.parametrize("musl", [0, 1])
@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED])
def test_nan_coordinate(dim, axis, deg, musl, prec):
    sc = cases.apply(cases.block(dim, deg, n=6 if dim == 3 else 12), use_musl=musl, flip_ratio=-0.95, precision=prec,
                     **cases.MODEL_CASES["dp"])
    sc = cases.box_plates(sc, BC.SlipFree, 0.3)
    _check(sc, sc.Np // 2, axis, np.nan)


@pytest.mark.parametrize("dim,axis", [(2, 0), (2, 1), (3, 0), (3, 1), (3, 2)])
@pytest.mark.parametrize("value", [np.nan, -np.inf, -1e300, -1e12])
@pytest.mark.parametrize("prec", [PREC_FP64, PREC_MIXED])
def test_lost_particle_of_a_periodic_scene(dim, axis, value, prec):
    """The grid of a periodic scene does not follow the particles."""
    sc = cases.apply(cases.periodic(dim), precision=prec)
    inner = np.all((sc.x > 0.02) & (sc.x < np.array([0.06, 0.08, 0.06])[:dim]), axis=1)
    near = inner & (sc.x[:, 0] < 3.0 * sc.params.dx)  # with a copy beyond x = Lx
    _check(sc, int(np.flatnonzero(near)[0]), axis, value)
