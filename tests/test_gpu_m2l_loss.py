"""FP64 M2L of sources whose low orders vanish (csrc/m2l_tc64.cuh k_m2l_pairs64):
dipoles or quadrupoles alone in fine cells, targets in coarse and distant ones,
where a fixed-point product would lose bits to its scales.  The targets have no
multipoles and no near sources, so their field is the far field alone; compared
with the products on the FP64 pipe (FMM_GB300_M2L_PRODUCT=cuda; their operators
fit shared memory to order 11).  Bar: 1e-14, FP64 sums of up to 144 terms a few
times larger than their total (a pair: 12 x 2^-53 x 4 = 5e-15), and less in the sum
over pairs."""
import numpy as np
import pytest

import fmm_gb300
import oracle
from fmm_gb300 import Options

pytestmark = pytest.mark.gpu


def _system(order, seed, m=2):
    rng = np.random.default_rng(seed)
    src = rng.uniform(-1.0, 1.0, (3000, 3))
    tgt = rng.uniform(-40.0, 40.0, (1500, 3))
    tgt = tgt[np.linalg.norm(tgt, axis=1) > 12.0]
    X = np.asfortranarray(np.concatenate([src, tgt]))
    M = np.zeros((len(X), fmm_gb300.n_components(m)), order="F")
    lo = fmm_gb300.n_components(order - 1) if order else 0
    M[:3000, lo:fmm_gb300.n_components(order)] = rng.normal(size=(3000, fmm_gb300.n_components(order) - lo))
    return X, M, np.arange(1, len(X) + 1, dtype=np.int32)[:, None]


@pytest.mark.parametrize("order", [0, 1, 2])
@pytest.mark.parametrize("p,theta", [(4, 0.5), (7, 0.4), (10, 0.3), (11, 0.5)])
def test_low_orders_vanish(order, p, theta, monkeypatch):
    X, M, E = _system(order, 10 * p + order)
    args = (0, X, M, E, theta, 8, p, 1)
    G = fmm_gb300.field_fmm(*args, options=Options.exact())
    assert fmm_gb300.last_stats()["t_m2l_product"] > 0.0
    monkeypatch.setenv("FMM_GB300_M2L_PRODUCT", "cuda")
    C = fmm_gb300.field_fmm(*args, options=Options.exact())
    far = slice(3000, None)
    for c in (slice(0, 1), slice(1, 4)):
        assert np.linalg.norm(G[far, c] - C[far, c]) <= 1e-14 * np.linalg.norm(C[far, c])


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("p", [5, 6])
def test_reference_tensors(order, p):
    """The reference's tensors (in the reduced basis and over all components).
    Bar: 1e-12, the FP64 path's against the oracle."""
    X, M, E = _system(order, p)
    args = (0, X, M, E, 0.5, 8, p, 1)
    G = fmm_gb300.field_fmm(*args)
    O = oracle.field_fmm(*args)
    far = slice(3000, None)
    assert np.linalg.norm(G[far] - O[far]) <= 1e-12 * np.linalg.norm(O[far])
