"""Rounding of the FP32 near field's potentials alone (csrc/near_f32.cu fold_of):
rms error of 24 systems of 700 points, every pair near, against the FP64 direct
sum.  Bars: the errors of sums folded at every leaf's end and fourth pair, one
hundredth above: these sums are the larger part of the error."""
import numpy as np
import pytest

import fmm_gb300
from fmm_gb300 import Options

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,damp,m,bar", [(3.0, "THOLE", 2, 7.45e-7), (20.0, "THOLE", 1, 1.81e-7),
                                              (20.0, "THOLE", 2, 3.07e-7), (20.0, "", 2, 1.37e-7),
                                              (200.0, "THOLE", 2, 1.85e-7)])
def test_rms(scale, damp, m, bar):
    err = []
    for seed in range(24):
        rng = np.random.default_rng(100 * seed + 10 * m)
        n = 700
        X = np.asfortranarray(rng.uniform(0.0, scale, (n, 3)))
        M = np.asfortranarray(rng.normal(size=(n, fmm_gb300.n_components(m))))
        E = np.arange(1, n + 1, dtype=np.int32)[:, None]
        d = rng.uniform(0.3, 0.8, n)
        G = fmm_gb300.field_fmm(0, X, M, E, 0.03, 24, 2, 0, damp, d, options=Options.exact(precision="mixed"))
        assert fmm_gb300.last_stats()["m2l_pairs"] == 0
        F = fmm_gb300.field_direct(0, X, M, E, 0, damp, d, options=Options.exact())
        err.append(np.linalg.norm(G - F) / np.linalg.norm(F))
    assert np.sqrt(np.mean(np.square(err))) <= bar
