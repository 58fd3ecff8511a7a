"""TF32 M2L products over the displacements of all eight octants at once
(csrc/m2l_gemm.cu, `mirrored`) against the CUDA-core products or per-pair
kernel, which know no octants.  Bars: those of the same comparison on larger
groups, twice the error of two FP32 products (2e-6) and the mixed path's
against FP64 (5e-6)."""
import numpy as np
import pytest

import fmm_gb300
from fmm_gb300 import Options
from helpers import rel_err

pytestmark = pytest.mark.gpu


def _system(kind, n, seed):
    rng = np.random.default_rng(seed)
    if kind == "blobs":
        cen, sig = rng.uniform(0.0, 90.0, (8, 3)), rng.uniform(2.0, 8.0, 8)
        k = rng.integers(0, 8, n)
        X = cen[k] + sig[k, None] * rng.normal(size=(n, 3))
    else:  # two sheets: displacements with zero components
        X = rng.uniform(0.0, 60.0, (n, 3))
        X[: n // 2, 2] = 30.0
        X[n // 2:, 0] = 10.0
    M = rng.normal(size=(n, 10)) * np.repeat([0.5, 0.1, 0.05], [1, 3, 6])
    return (0, np.asfortranarray(X), np.asfortranarray(M), np.arange(1, n + 1, dtype=np.int32)[:, None])


@pytest.mark.parametrize("kind", ["blobs", "planes"])
@pytest.mark.parametrize("p", [1, 2, 7, 10, 11, 12])
def test_mirrored_groups(kind, p, monkeypatch):
    args = _system(kind, 3001, p)
    mixed = Options.exact(precision="mixed")
    F64 = fmm_gb300.field_fmm(*args, 0.5, 16, p, 2, "", options=Options.exact())
    F = fmm_gb300.field_fmm(*args, 0.5, 16, p, 2, "", options=mixed)
    s = fmm_gb300.last_stats()
    monkeypatch.setenv("FMM_GB300_M2L_PRODUCT", "cuda")
    C = fmm_gb300.field_fmm(*args, 0.5, 16, p, 2, "", options=mixed)
    groups = fmm_gb300.last_stats()["m2l_groups"]
    assert 0 < s["m2l_groups"] < groups <= 8 * s["m2l_groups"]
    assert np.all(np.isfinite(F))
    assert rel_err(F, C) < 2e-6
    assert rel_err(F, F64) < 5e-6
