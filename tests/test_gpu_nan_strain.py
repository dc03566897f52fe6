"""A particle whose deformation gradient is not a number keeps that state through
the return mapping, as in the reference (std::max(sigma, 1e-4) is NaN there): no
model projects it to a finite one.

Against the oracle, in which the NaN force reaches every particle of a small
block: the same entries are NaN, and the scalars that a model leaves alone are
the same ones (1e-10 of their size, as in the other one-step parity tests)."""
import numpy as np
import pytest

import cases
from gpu_util import needs_gpu, run_gpu, run_oracle

pytestmark = [pytest.mark.gpu, needs_gpu]


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("musl", [0, 1])
@pytest.mark.parametrize("model", ["mcc_nohard", "mcc_expoexpl", "mcc_expoimpl", "mcc_sinhimpl", "mccvisc", "mccmui_expoimpl",
                                   "dp", "dpsoft", "dpmui", "vm", "vmvisc_capped", "noplast"])
def test_nan_strain_stays_nan(dim, musl, model):
    sc = cases.apply(cases.block(dim, 3, n=4), use_musl=musl, **cases.MODEL_CASES[model])
    sc.F[sc.Np // 2] = np.nan
    g, o = run_gpu(sc, 1), run_oracle(sc, 1)
    assert not np.any(np.isfinite(o["p"]["F"]))
    assert not np.any(np.isfinite(g["p"]["F"]))
    a, b = g["p"]["scalars"], o["p"]["scalars"]
    np.testing.assert_array_equal(np.isfinite(a), np.isfinite(b))
    kept = np.isfinite(b)
    np.testing.assert_allclose(a[kept], b[kept], rtol=1e-10, atol=0.0)
