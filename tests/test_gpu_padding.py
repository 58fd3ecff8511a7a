"""The packed FP32 near field's padding of odd leaves (csrc/near_f32.cu
k_gather_x2): particles on regular positions, among them places 1000 from a
leaf's last particle, at twice its coordinate and at the root's plane.  A target
that met the empty particle would have 0 x infinity in its field.  Bar: the mixed
path's against FP64 (5e-6)."""
import numpy as np
import pytest

import fmm_gb300
from fmm_gb300 import Options
from helpers import rel_err

pytestmark = pytest.mark.gpu


def _chain(n, pitch):
    X = np.zeros((n, 3))
    X[:, 0] = pitch * np.arange(n)
    return X


def _lattice(k, pitch):
    g = pitch * np.arange(k)
    return np.stack(np.meshgrid(g, g, g, indexing="ij"), axis=-1).reshape(-1, 3)


SYSTEMS = {
    "chain": _chain(1000, 10.0),             # padding of a leaf of 63 at +1000: a particle's place
    "long_chain": _chain(601, 250.0),        # beyond 1000 from the centre
    "lattice": _lattice(9, 125.0),           # root centre on a particle
    "wide_lattice": _lattice(9, 1000.0),
    "even_lattice": _lattice(10, 500.0),
}


@pytest.mark.parametrize("kind", sorted(SYSTEMS))
@pytest.mark.parametrize("m,f,damp", [(0, 0, ""), (2, 1, ""), (2, 1, "AMOEBA"), (1, 1, "ERF")])
def test_regular_positions(kind, m, f, damp):
    X = np.asfortranarray(SYSTEMS[kind])
    n = X.shape[0]
    rng = np.random.default_rng(n)
    M = np.asfortranarray(rng.uniform(0.2, 1.0, (n, fmm_gb300.n_components(m))))
    E = np.arange(1, n + 1, dtype=np.int32)[:, None]
    d = rng.uniform(0.4, 0.8, n)
    for ncrit in (5, 64):
        args = (0, X, M, E, 0.5, ncrit, 6, f, damp, d)
        G = fmm_gb300.field_fmm(*args, options=Options.exact(precision="mixed"))
        assert fmm_gb300.last_stats()["p2p_particle_pairs"] > 0
        F = fmm_gb300.field_fmm(*args, options=Options.exact())
        assert np.all(np.isfinite(G))
        assert rel_err(G, F) < 5e-6
