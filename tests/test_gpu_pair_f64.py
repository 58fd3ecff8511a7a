"""The FP64 pair kernels (csrc/near.cu, csrc/pair_f64.cuh) against the CPU
oracle at the sizes where their layout changes: steps of 32 sources and their
remainders, slices of the source list, exclusion lists longer than the
registers hold, and pair distances on both sides of the damping cut-off.
Bar: 1e-12, the FP64 path's."""
import numpy as np
import pytest

import fmm_gb300
import oracle
from fmm_gb300 import Options
from helpers import rel_err, small_system

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _with_exclusions(s, width, seed):
    """Random partners (the particle itself first), unused slots between them
    and one entry twice."""
    n = s["coordinates"].shape[0]
    rng = np.random.default_rng(seed)
    E = rng.integers(0, n + 1, (n, width)).astype(np.int32)
    E[:, 0] = np.arange(1, n + 1)
    if width > 3:
        E[:, 2] = 0
        E[:, width - 1] = E[:, 1]
    s["exclusions"] = np.asfortranarray(E)
    return s


@pytest.mark.parametrize("n", [31, 32, 33, 65, 300, 1025])
@pytest.mark.parametrize("width", [1, 4, 5, 7])
@pytest.mark.parametrize("excl", ["ref", "mask"])
def test_direct_sizes(n, width, excl):
    m, f, damp = [(2, 2, "THOLE"), (2, 1, ""), (1, 2, "AMOEBA"), (3, 1, "ERF")][n % 4]
    s = _with_exclusions(small_system(n, 2.0 * n ** (1 / 3), order=m, seed=n, damp=damp), width, n + width)
    d = s["damping_factors"] if damp else None
    args = (0, s["coordinates"], s["multipoles"], s["exclusions"])
    G = fmm_gb300.field_direct(*args, f, damp, d, options=Options(excl_mode=excl))
    O = oracle.field_direct(*args, f, damp, d, excl_mode=excl)
    cols = slice(1, None) if damp == "AMOEBA" else slice(0, None)
    assert np.all(np.isfinite(G))
    assert rel_err(G, O, cols) <= TOL


@pytest.mark.parametrize("damp", ["THOLE", "AMOEBA", "ERF"])
@pytest.mark.parametrize("mf", [(0, 0), (2, 2), (3, 3)])
def test_damping_cutoff(damp, mf):
    """Each source alone at a distance on either side of every switch of the
    damped kernels; per target, in the order-f components."""
    m, f = mf
    a = 0.5
    r = np.concatenate([np.geomspace(0.05, 5.0, 12), np.linspace(5.0, 260.0, 53)])
    for k, x in enumerate(r):
        X = np.asfortranarray(np.array([[0.0, 0.0, 0.0], [0.48 * x, -0.6 * x, 0.64 * x]]))
        M = np.asfortranarray(np.random.default_rng(k).uniform(0.1, 1.0, (2, fmm_gb300.n_components(m))))
        E = np.asfortranarray(np.array([[1], [2]], dtype=np.int32))
        d = np.full(2, a ** 0.5)
        G = fmm_gb300.field_direct(0, X, M, E, f, damp, d, options=Options(excl_mode="mask"))
        O = oracle.field_direct(0, X, M, E, f, damp, d, excl_mode="mask")
        # each order against the magnitude of its own components: the tensor
        # components of one order have the size (2k - 1)!! / r^(k + 1) before
        # any cancellation among the sources' orders
        for k0, k1 in zip((0, 1, 4, 10), (1, 4, 10, 20)):
            if k1 > G.shape[1]:
                break
            scale = max(np.max(np.abs(O[:, k0:k1])), np.finfo(float).tiny)
            assert np.max(np.abs(G[:, k0:k1] - O[:, k0:k1])) <= 1e-11 * scale, (x, k0)


@pytest.mark.parametrize("n,ncrit", [(40, 8), (333, 16), (2500, 64), (12000, 64)])
@pytest.mark.parametrize("coef", ["ref", "exact"])
def test_near_field_slices(n, ncrit, coef):
    damp = "AMOEBA" if n % 2 else "THOLE"
    s = _with_exclusions(small_system(n, 2.0 * n ** (1 / 3), order=2, seed=n, damp=damp), 6, n)
    args = (0, s["coordinates"], s["multipoles"], s["exclusions"], 0.5, ncrit, 4, 2, damp, s["damping_factors"])
    excl = "ref" if coef == "ref" else "mask"
    G = fmm_gb300.field_fmm(*args, options=Options(coef_mode=coef, excl_mode=excl))
    O = oracle.field_fmm(*args, coef_mode=coef, excl_mode=excl)
    cols = slice(1, None) if damp == "AMOEBA" else slice(0, None)
    assert rel_err(G, O, cols) <= TOL
