"""The mixed form's node offsets x_i - x_p are FP64 differences rounded once.

dx is chosen a little under half an FP32 ulp above a representable number, so
that offsets formed in FP32 from a rounded dx come out 5.8e-8 too short, all of
them.  Lone particles with an affine velocity B and no stress show the offsets in
three places: the node velocities of the P2G, the B of the gather and the node
velocities of the MUSL re-scatter.

Rounding to nearest has no preferred sign: a value takes at most about eight
roundings of 2^-25 rms or less (8e-8 together), and the mean over 200 or more
independent offsets stays within 1.5e-8, more than twice its standard error.
The largest single error is bounded by twelve roundings of 2^-24."""
import numpy as np
import pytest

from matter_tests_b200.abi import PREC_MIXED

import cases
from gpu_util import needs_gpu, run_gpu

pytestmark = [pytest.mark.gpu, needs_gpu]

DX = 0.0078125 * (1.0 + 0.98 * 2.0 ** -24)
MEAN, WORST = 1.5e-8, 12 * 2.0 ** -24
F32 = np.float32


def _lone_particles(dim, deg, musl):
    per = 6 if dim == 3 else 16
    sc = cases.apply(cases.block(dim, deg, n=6 if dim == 3 else 12), use_musl=musl, flip_ratio=-2.0, precision=PREC_MIXED,
                     plastic_model=cases.PM.NoPlasticity, gravity=(0.0, 0.0, 0.0), dx=DX)
    rng = np.random.default_rng(8)
    cells = np.stack(np.meshgrid(*[8.0 * np.arange(per)] * dim, indexing="ij"), -1).reshape(-1, dim)
    n = len(cells)
    sc.x = (cells + rng.uniform(0.0, 1.0, size=(n, dim))) * DX
    sc.v = np.zeros((n, dim))
    sc.B = np.zeros((n, dim, dim))
    for a in range(dim):
        sc.B[:, a, a] = rng.uniform(1.0, 2.0, size=n) * DX ** 2
    sc.F = sc.scalars = None
    sc.plates, sc.objects = [], []
    return sc


def _stencils(sc, g):
    """Per particle: the flat indices of its 4^dim nodes and their offsets, in FP64."""
    dim = sc.dim
    axes = [g["g"][k] for k in "xyz"[:dim]]
    N = g["g"]["dims"]
    flat, off = np.zeros((len(sc.x),) + (1,) * dim, dtype=np.int64), []
    for a in range(dim):
        base = np.floor((sc.x[:, a] - axes[a][0]) / DX).astype(np.int64) - 1
        i = base[:, None] + np.arange(4)
        shape = (len(sc.x),) + tuple(4 if b == a else 1 for b in range(dim))
        stride = int(np.prod(N[a + 1:dim])) if a + 1 < dim else 1
        flat = flat + (i * stride).reshape(shape)
        off.append((axes[a][i] - sc.x[:, a, None]).reshape(shape))
    off = [np.broadcast_to(o, flat.shape).reshape(len(sc.x), -1) for o in off]
    return flat.reshape(len(sc.x), -1), np.stack(off, -1)


def _affine(sc, B, off, deg):
    """B D^-1 (x_i - x_p) with the FP32 products that the kernels stage; B column-major."""
    apic = F32(3.0 / DX ** 2) if deg == 3 else F32(4.0 / DX ** 2)
    q = (apic * B.astype(F32)).astype(np.float64).transpose(0, 2, 1)
    return np.einsum("pab,pnb->pna", q, off)


def _check(rel, what):
    assert len(rel) >= 200
    assert np.abs(rel).max() <= WORST, (what, np.abs(rel).max())
    assert abs(rel.mean()) <= MEAN, (what, rel.mean())


@pytest.mark.parametrize("dim,deg", [(2, 2), (2, 3), (3, 2), (3, 3)])
def test_p2g_and_gather(dim, deg):
    sc = _lone_particles(dim, deg, 0)
    g = run_gpu(sc, 1)
    flat, off = _stencils(sc, g)
    v, m = g["g"]["v"][flat], g["g"]["mass"][flat]
    want = _affine(sc, sc.B.reshape(-1, dim, dim), off, deg)
    big = (m > 1e-6 * m.max())[..., None] & (np.abs(off) > 0.05 * DX)
    _check((v / np.where(big, want, 1.0) - 1.0)[big], "P2G")
    u = np.abs(off) / DX
    if deg == 3:  # the spline with its FP32 constants, which are a little large
        w = np.where(u < 1, 0.5 * u ** 3 - u ** 2 + float(F32(2 / 3)),
                     np.where(u < 2, float(F32(1 / 6)) * (2 - u) ** 3, 0.0)).prod(-1)
    else:
        w = np.where(u < 0.5, 0.75 - u ** 2, np.where(u < 1.5, 0.5 * (1.5 - u) ** 2, 0.0)).prod(-1)
    B = np.einsum("pn,pna,pnb->pab", w, v, off)
    got = g["p"]["B"].reshape(-1, dim, dim)
    rel = np.stack([got[:, a, a] / B[:, a, a] - 1.0 for a in range(dim)])
    _check(rel.reshape(-1), "gather")


@pytest.mark.parametrize("dim,deg", [(2, 2), (2, 3), (3, 2), (3, 3)])
def test_musl_rescatter(dim, deg):
    sc = _lone_particles(dim, deg, 1)
    g = run_gpu(sc, 1)
    flat, off = _stencils(sc, g)
    v, m = g["g"]["v"][flat], g["g"]["mass"][flat]
    want = g["p"]["v"][:, None, :] + _affine(sc, g["p"]["B"].reshape(-1, dim, dim), off, deg)
    big = (m > 1e-6 * m.max())[..., None] & (np.abs(off) > 0.2 * DX)
    _check((v / np.where(big, want, 1.0) - 1.0)[big], "re-scatter")
