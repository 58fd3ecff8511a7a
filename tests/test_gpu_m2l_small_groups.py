"""Mixed calls whose displacement groups hold few pairs (csrc/m2l_gemm.cu
kMinGroupPairs): summed in FP64, not in TF32 parts with the octants' groups joined.
Their error against the FP64 call is no larger than that of the per-pair kernel,
which takes such groups beside the CUDA-core products (and which is FP64 above
order 8; 1.1 for the order of the sums)."""
import numpy as np
import pytest

import fmm_gb300
from fmm_gb300 import Options, Plan
from helpers import rel_err

pytestmark = pytest.mark.gpu


def _args(p, f=1):
    rng = np.random.default_rng(1)
    cen, sig = rng.uniform(0.0, 90.0, (8, 3)), rng.uniform(2.0, 8.0, 8)
    k = rng.integers(0, 8, 3001)
    X = np.asfortranarray(cen[k] + sig[k, None] * rng.normal(size=(3001, 3)))
    M = np.asfortranarray(rng.normal(size=(3001, 10)) * np.repeat([0.5, 0.1, 0.05], [1, 3, 6]))
    return (0, X, M, np.arange(1, 3002, dtype=np.int32)[:, None], 0.5, 16, p, f)


@pytest.mark.parametrize("p", [3, 6, 8, 9, 12])
def test_error(p, monkeypatch):
    args = _args(p)
    opt = Options.exact(precision="mixed_far")
    F = fmm_gb300.field_fmm(*args, options=Options.exact())
    G = fmm_gb300.field_fmm(*args, options=opt)
    assert fmm_gb300.last_stats()["t_m2l_product"] > 0.0
    monkeypatch.setenv("FMM_GB300_M2L_PRODUCT", "cuda")
    C = fmm_gb300.field_fmm(*args, options=opt)
    s = fmm_gb300.last_stats()
    assert s["m2l_pairs"] < 16 * s["m2l_groups"] and s["t_m2l_product"] <= 0.0
    field = slice(1, 4)
    assert rel_err(G, F, field) <= 1.1 * rel_err(C, F, field)


def test_plan():
    """Replays keep the FP64 products."""
    args = _args(7)
    opt = Options.exact(precision="mixed")
    plan = Plan(args[1], 10, args[3], 0.5, 16, 7, 1, options=opt)
    for scale in (1.0, -2.0):
        F = plan.execute(np.asfortranarray(scale * args[2]))
        G = fmm_gb300.field_fmm(0, args[1], scale * args[2], *args[3:], options=opt)
        assert rel_err(F, G) <= 1e-12
