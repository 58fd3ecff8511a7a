"""The FP64 grouped M2L (csrc/m2l_tc64.cuh: fixed-point products on the tensor
cores) against the CPU oracle: expansion orders on both sides of the operator's
128-row parts and of its chunks of 16 components, in the reduced basis and (ref
mode above order 5) over all Cartesian components; group sizes that do and do
not fill a task; multipoles of any magnitude and non-finite ones.  Thole damping
keeps the near pairs from dominating the norm.  Bar: 1e-12, the FP64 path's."""
import os

import numpy as np
import pytest

import fmm_gb300
import oracle
from fmm_gb300 import Options, systems
from helpers import rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _args(s, theta, ncrit, p, f=1):
    return (0, s["coordinates"], s["multipoles"], s["exclusions"], theta, ncrit, p, f, "THOLE", s["damping_factors"])


@pytest.mark.parametrize("p", [0, 1, 3, 4, 7, 10, 11, 12])
def test_reduced_basis(p):
    s = systems.water(700, 35.0, seed=p)
    kw = dict(coef_mode="exact", excl_mode="mask")
    G = fmm_gb300.field_fmm(*_args(s, 0.5, 32, p), options=Options(**kw))
    assert fmm_gb300.last_stats()["m2l_groups"] > 0
    O = oracle.field_fmm(*_args(s, 0.5, 32, p), **kw)
    assert rel_err(G, O) <= TOL


@pytest.mark.parametrize("p", [5, 6, 7, 8, 10])
def test_reference_tensors(p):
    """int32 coefficients: exact to order 5, wrapped above (the wrapped
    tensors' sums are orders of magnitude off the true field)."""
    s = systems.water(500, 32.0, seed=20 + p)
    G = fmm_gb300.field_fmm(*_args(s, 0.5, 32, p))
    O = oracle.field_fmm(*_args(s, 0.5, 32, p))
    assert rel_err(G, O) <= TOL


@pytest.mark.parametrize("n_mol,ncrit", [(60, 8), (333, 12), (2001, 40)])
def test_group_sizes(n_mol, ncrit):
    s = systems.water(n_mol, (59.05 * n_mol) ** (1 / 3), seed=n_mol)
    for mode in ("ref", "exact"):
        kw = dict(coef_mode=mode, excl_mode="ref" if mode == "ref" else "mask")
        G = fmm_gb300.field_fmm(*_args(s, 0.6, ncrit, 4, 2), options=Options(**kw))
        O = oracle.field_fmm(*_args(s, 0.6, ncrit, 4, 2), **kw)
        assert rel_err(G, O) <= TOL


@pytest.mark.parametrize("scale", [1e-200, 1e-24, 1e20, 1e180])
def test_magnitudes(scale):
    """Power-of-two scales follow the operands: same relative result at any
    magnitude."""
    s = systems.water(400, 29.0, seed=5)
    kw = dict(coef_mode="exact", excl_mode="mask")
    s["multipoles"] = s["multipoles"] * scale
    G = fmm_gb300.field_fmm(*_args(s, 0.5, 32, 8), options=Options(**kw))
    O = oracle.field_fmm(*_args(s, 0.5, 32, 8), **kw)
    assert rel_err(G / scale, O / scale) <= TOL


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_multipoles(bad):
    s = systems.water(400, 29.0, seed=6)
    s["multipoles"][37, 0] = bad
    G = fmm_gb300.field_fmm(*_args(s, 0.5, 32, 6), options=Options(coef_mode="exact", excl_mode="mask"))
    far = np.delete(np.arange(G.shape[0]), [36, 37, 38])
    assert not np.any(np.isfinite(G[far, 0]))


def test_products_agree():
    """Tensor cores against the FP64 pipe (FMM_GB300_M2L_PRODUCT=cuda)."""
    s = systems.water(3000, 56.0, seed=8)
    opt = Options(coef_mode="exact", excl_mode="mask")
    G = fmm_gb300.field_fmm(*_args(s, 0.4, 64, 9), options=opt)
    os.environ["FMM_GB300_M2L_PRODUCT"] = "cuda"
    try:
        C = fmm_gb300.field_fmm(*_args(s, 0.4, 64, 9), options=opt)
    finally:
        del os.environ["FMM_GB300_M2L_PRODUCT"]
    # both round at 2^-53 of sums of about a hundred terms per pair
    assert rel_err(G, C) <= 1e-13
