"""ERF damping in the FP32 near-field kernels (csrc/near_f32.cu), pair by pair,
against the CPU oracle: three particles in as many leaves (a cell of ncrit = 2 is
split; systems of no more particles than ncrit are summed directly in FP64), the
third without multipoles, a r^2 over every interval of
the Boys table and both sides of the far switches (24, 28, 32 for up to 2, 4 and
more derivatives), packed and one-source kernels.  Bar: 2e-6 of the source
components' own fields, some thirty FP32 roundings: the displacement's and
r^-(2j+1)'s errors up to the ninth power of r, the polynomial, the recursion."""
import numpy as np
import pytest

import fmm_gb300
import oracle
from fmm_gb300 import Options

pytestmark = pytest.mark.gpu

S = np.concatenate([np.geomspace(1e-4, 0.9, 8), np.arange(0.99, 34.0, 0.5), [23.999, 24.001, 27.999, 28.001, 60.0]])
A = 0.3
E = np.asfortranarray(np.array([[1], [2], [3]], dtype=np.int32))


def _pair(k, r, m):
    X = np.asfortranarray(r * np.array([[0.0, 0.0, 0.0], [0.48, -0.6, 0.64], [0.9, 0.2, 0.1]]))
    M = np.random.default_rng(k).uniform(0.1, 1.0, (3, fmm_gb300.n_components(m)))
    M[2] = 0.0
    return X, np.asfortranarray(M)


@pytest.mark.parametrize("mf", [(0, 0), (1, 0), (0, 1), (1, 1), (2, 1), (0, 2), (2, 2)])
@pytest.mark.parametrize("packed", ["1", "0"])
def test_erf_pairs(mf, packed, monkeypatch):
    monkeypatch.setenv("FMM_GB300_P2P_PACKED", packed)
    m, f = mf
    d = np.full(3, A ** 0.5)
    same = 0
    for k, r in enumerate(np.sqrt(S / A)):
        X, M = _pair(k, r, m)
        args = (0, X, M, E, 0.5, 2, 4, f, "ERF", d)
        G = fmm_gb300.field_fmm(*args, options=Options.exact(precision="mixed"))
        st = fmm_gb300.last_stats()
        assert st["num_leaves"] == 3 and st["p2p_particle_pairs"] == 9 and st["m2l_pairs"] == 0
        F = fmm_gb300.field_fmm(*args, options=Options.exact())
        same += np.array_equal(G, F)
        O = oracle.field_direct(0, X, M, E, f, "ERF", d, excl_mode="mask")
        terms = 0.0  # magnitudes of the source components' own fields, which may cancel in the sum
        for c in range(M.shape[1]):
            Mc = np.zeros_like(M)
            Mc[:, c] = M[:, c]
            terms = terms + np.abs(oracle.field_direct(0, X, Mc, E, f, "ERF", d, excl_mode="mask"))
        for o in range(f + 1):
            c = slice(fmm_gb300.n_components(o - 1) if o else 0, fmm_gb300.n_components(o))
            err = np.linalg.norm(G[:2, c] - O[:2, c]) / np.linalg.norm(terms[:2, c])
            assert err <= 2e-6, (S[k], o, err)
            assert np.linalg.norm(F[:2, c] - O[:2, c]) <= 1e-13 * np.linalg.norm(terms[:2, c])
    assert same == 0  # the FP64 kernels did not run in the FP32 ones' place


@pytest.mark.parametrize("mf", [(1, 1), (2, 2)])
@pytest.mark.parametrize("bad", [-0.5, np.nan])
def test_factors_out_of_range(mf, bad):
    """Factors of both signs and NaN: NaN in the pair, as the root of a is."""
    m, f = mf
    X, M = _pair(1, 1.2, m)
    G = fmm_gb300.field_fmm(0, X, M, E, 0.5, 2, 4, f, "ERF", np.array([0.6, bad, 0.6]),
                            options=Options.exact(precision="mixed"))
    assert np.all(np.isnan(G[:2]))
