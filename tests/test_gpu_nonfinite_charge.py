"""Infinite and NaN charges under AMOEBA damping in the FP64 pair kernels
(csrc/pair_f64.cuh): the damped potential has no charge term, 0 x charge, which
such a charge makes NaN in every other particle's potential as in the oracle's."""
import numpy as np
import pytest

import fmm_gb300
import oracle
from fmm_gb300 import Options
from helpers import small_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("mf", [(0, 0), (1, 1), (2, 1), (2, 2), (3, 1)])
@pytest.mark.parametrize("how", ["direct", "near"])
def test_amoeba(bad, mf, how):
    m, f = mf
    s = small_system(40, 8.0, order=m, seed=m + f, damp="AMOEBA")
    s["multipoles"][7, 0] = bad
    E = np.arange(1, 41, dtype=np.int32)[:, None]
    args = (0, s["coordinates"], s["multipoles"], E)
    d = s["damping_factors"]
    opt = Options(coef_mode="exact", excl_mode="mask")
    if how == "direct":
        G = fmm_gb300.field_direct(*args, f, "AMOEBA", d, options=opt)
    else:
        G = fmm_gb300.field_fmm(*args, 0.05, 16, 2, f, "AMOEBA", d, options=opt)  # every pair is near
        assert fmm_gb300.last_stats()["m2l_pairs"] == 0
    O = oracle.field_direct(*args, f, "AMOEBA", d, excl_mode="mask")
    assert np.array_equal(np.isfinite(G), np.isfinite(O))  # (a gradient's diagonal: two infinite terms, NaN)
    assert np.array_equal(np.isnan(G[:, :4]), np.isnan(O[:, :4]))
    others = np.delete(np.arange(40), 7)
    assert np.all(np.isnan(G[others, 0])) and np.all(np.isfinite(G[7]))
