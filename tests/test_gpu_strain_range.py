"""The return mapping over the whole range of strains: the series of the Hencky
strain changes its degree with the strain and hands strains beyond about 10% to
the singular value decomposition, and a particle may be rotated by any angle.

Each case is one step against the oracle.  Tolerance: as the other one-step
parity tests (1e-10 of each field's scale, plus 100x the oracle's own spread
under a few-ulp perturbation): the series are cut below FP64 rounding.
"""
import numpy as np
import pytest

from matter_tests_b200.abi import BC

import cases
from gpu_util import compare_states, needs_gpu, oracle_sensitivity, run_gpu, run_oracle

pytestmark = [pytest.mark.gpu, needs_gpu]

# strain amplitudes on both sides of every change of degree and of the hand-over
AMPLITUDES = [0.0, 1e-12, 1e-4, 1.5e-3, 3e-3, 9e-3, 2e-2, 4e-2, 9e-2, 0.12, 0.25]


def _scene(dim, model, amp, rotate, seed=5):
    sc = cases.apply(cases.block(dim, 2, n=4 if dim == 3 else 7, seed=seed), **cases.MODEL_CASES[model])
    sc = cases.box_plates(sc, BC.SlipFree, 0.3)
    rng = np.random.default_rng(seed + 10)
    n = sc.Np
    F = np.eye(dim) + rng.uniform(-amp, amp, size=(n, dim, dim))
    if rotate:
        q, _ = np.linalg.qr(rng.normal(size=(n, dim, dim)))
        q[np.linalg.det(q) < 0, :, 0] *= -1
        F = F @ q
    sc.F = np.ascontiguousarray(np.transpose(F, (0, 2, 1)))
    return sc


@pytest.mark.parametrize("rotate", [False, True])
@pytest.mark.parametrize("amp", AMPLITUDES)
@pytest.mark.parametrize("dim,model", [(3, "dp"), (3, "dpmui"), (3, "vm"), (3, "noplast"), (2, "dp"), (2, "vmvisc_capped")])
def test_strain_range_one_step(dim, model, amp, rotate):
    sc = _scene(dim, model, amp, rotate)
    g, o = run_gpu(sc, 1), run_oracle(sc, 1)
    compare_states(g, o, 1e-10, sens=oracle_sensitivity(sc, 1))


@pytest.mark.parametrize("model", ["dp_cohesion", "dpvisc"])
def test_projection_to_a_far_tip_is_applied_in_parts(model):
    """A cohesion of the size of the bulk modulus moves the tip to strains of order one."""
    sc = _scene(3, model, 5e-2, False)
    sc.params.q_cohesion = -1.5 * sc.params.E
    g, o = run_gpu(sc, 1), run_oracle(sc, 1)
    compare_states(g, o, 1e-10, sens=oracle_sensitivity(sc, 1))
