"""M2M and L2L with one, two and four children at a time (csrc/translate.cu):
orders on both sides of the switches and nodes with one to eight children,
against the CPU oracle (FP64, 1e-12) and the FP64 path (mixed, 5e-6)."""
import numpy as np
import pytest

import fmm_gb300
import oracle
from fmm_gb300 import Options
from helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [0, 1, 6, 7, 8, 9, 10])
@pytest.mark.parametrize("shape", ["cube", "rod"])
def test_child_groups(p, shape):
    rng = np.random.default_rng(p)
    n = 1500
    X = rng.uniform(0.0, 30.0, (n, 3))
    if shape == "rod":  # nodes of one or two children beside full ones
        X[:, 1:] *= 0.05
        X[: n // 2, 1:] += rng.uniform(0.0, 20.0, 2)
    X = np.asfortranarray(X)
    M = np.asfortranarray(rng.normal(size=(n, 4)))
    E = np.arange(1, n + 1, dtype=np.int32)[:, None]
    args = (0, X, M, E, 0.5, 8, p, 1, "")
    F = fmm_gb300.field_fmm(*args, options=Options(coef_mode="exact", excl_mode="mask"))
    O = oracle.field_fmm(*args, coef_mode="exact", excl_mode="mask")
    assert rel_err(F, O) <= 1e-12
    G = fmm_gb300.field_fmm(*args, options=Options(coef_mode="exact", excl_mode="mask", precision="mixed"))
    assert rel_err(G, F) <= 5e-6
