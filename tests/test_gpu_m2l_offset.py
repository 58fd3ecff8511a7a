"""Far-field pairs of systems far from the origin (csrc/m2l_gemm.cu
kGroupDeviation): cell centres are rounded at the coordinates' size, and a group's
common displacement is off a pair's own by it.  Reference-mode calls and those of
small groups take each pair's own there.  Bar: the FP64 path's against the oracle,
1e-12."""
import numpy as np
import pytest

import fmm_gb300
import oracle
from fmm_gb300 import Options
from helpers import rel_err

pytestmark = pytest.mark.gpu


def _system(offset, n, seed, m):
    rng = np.random.default_rng(seed)
    X = np.asfortranarray(rng.uniform(0.0, 3.0, (n, 3)) + offset * np.array([1.0, -0.7, 0.4]))
    M = np.asfortranarray(rng.normal(size=(n, fmm_gb300.n_components(m))))
    d = rng.uniform(0.4, 0.8, n)
    return X, M, np.arange(1, n + 1, dtype=np.int32)[:, None], d


@pytest.mark.parametrize("offset", [0.0, 30.0, 1.0e3, 1.0e4])
@pytest.mark.parametrize("p,m", [(4, 1), (5, 3), (7, 2)])
def test_reference_mode(offset, p, m):
    X, M, E, d = _system(offset, 1500, p, m)
    args = (0, X, M, E, 0.8, 6, p, 1, "THOLE", 0.1 * d)  # near pairs damped away
    G = fmm_gb300.field_fmm(*args)
    s = fmm_gb300.last_stats()
    assert s["m2l_pairs"] > 0
    if offset != 30.0:  # (near the line there)
        assert (s["t_m2l_product"] > 0.0) == (offset == 0.0)
    assert rel_err(G, oracle.field_fmm(*args)) <= 1e-12


@pytest.mark.parametrize("offset", [0.0, 1.0e4])
def test_small_groups(offset):
    X, M, E, d = _system(offset, 300, 3, 2)
    args = (0, X, M, E, 0.6, 8, 8, 1, "THOLE", 0.1 * d)
    G = fmm_gb300.field_fmm(*args, options=Options(coef_mode="exact", excl_mode="mask"))
    s = fmm_gb300.last_stats()
    assert 0 < s["m2l_pairs"] < 16 * s["m2l_groups"]
    assert rel_err(G, oracle.field_fmm(*args, coef_mode="exact", excl_mode="mask")) <= 1e-12
