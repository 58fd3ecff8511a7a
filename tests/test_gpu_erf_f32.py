"""FP32 near field with ERF damping (csrc/pair.cuh: Boys functions by interval
polynomials, undamped pairs beyond the tail) against the CPU oracle: one pair
at a time, over every interval and both sides of the far switches, per order of
the field.  Bar: 2e-6, some thirty FP32 roundings: the displacement's and
r^-(2j+1)'s errors up to the ninth power of r, the polynomial, the recursion."""
import numpy as np
import pytest

import fmm_gb300
import oracle
from fmm_gb300 import Options

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mf", [(0, 0), (1, 1), (2, 1), (2, 2), (3, 3)])
@pytest.mark.parametrize("packed", ["1", "0"])
def test_erf_pairs(mf, packed, monkeypatch):
    monkeypatch.setenv("FMM_GB300_P2P_PACKED", packed)
    m, f = mf
    a = 0.3
    s = np.concatenate([np.geomspace(1e-4, 0.9, 8), np.arange(0.99, 34.0, 0.5), [23.999, 24.001, 27.999, 28.001, 60.0]])
    E = np.asfortranarray(np.array([[1], [2]], dtype=np.int32))
    d = np.full(2, a ** 0.5)
    for k, r in enumerate(np.sqrt(s / a)):
        X = np.asfortranarray(np.array([[0.0, 0.0, 0.0], [0.48 * r, -0.6 * r, 0.64 * r]]))
        M = np.asfortranarray(np.random.default_rng(k).uniform(0.1, 1.0, (2, fmm_gb300.n_components(m))))
        G = fmm_gb300.field_fmm(0, X, M, E, 0.5, 64, 4, f, "ERF", d,
                                options=Options.exact(precision="mixed", excl_mode="mask"))
        O = oracle.field_direct(0, X, M, E, f, "ERF", d, excl_mode="mask")
        terms = 0.0  # magnitudes of the source components' own fields, which may cancel in the sum
        for c in range(M.shape[1]):
            Mc = np.zeros_like(M)
            Mc[:, c] = M[:, c]
            terms = terms + np.abs(oracle.field_direct(0, X, Mc, E, f, "ERF", d, excl_mode="mask"))
        for o in range(f + 1):
            c = slice(fmm_gb300.n_components(o - 1) if o else 0, fmm_gb300.n_components(o))
            err = np.linalg.norm(G[:, c] - O[:, c]) / np.linalg.norm(terms[:, c])
            assert err <= 2e-6, (s[k], o, err)
