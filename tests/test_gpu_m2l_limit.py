"""The grouped M2L's memory limit (csrc/m2l_gemm.cu grouped_bytes): where it is
reached, the pairs of reference-mode and periodic calls, and those of small
groups, go one by one, with the same result.  Bar: the FP64 path's, 1e-12."""
import numpy as np
import pytest

import fmm_gb300
import oracle
from fmm_gb300 import Options, systems
from helpers import potential_up_to_constant, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [3, 5, 6])
def test_reference_mode(p, monkeypatch):
    s = systems.water(400, 29.0, seed=p)
    args = (0, s["coordinates"], s["multipoles"], s["exclusions"], 0.5, 32, p, 1, "THOLE", s["damping_factors"])
    G = fmm_gb300.field_fmm(*args)
    g = fmm_gb300.last_stats()
    monkeypatch.setenv("FMM_GB300_M2L_BYTES", "1000")
    P = fmm_gb300.field_fmm(*args)
    assert g["t_m2l_product"] > 0.0 and fmm_gb300.last_stats()["t_m2l_product"] <= 0.0
    O = oracle.field_fmm(*args)
    assert rel_err(G, O) <= 1e-12 and rel_err(P, O) <= 1e-12


def test_periodic(monkeypatch):
    s = systems.water(120, 19.0, seed=3)
    box = np.asfortranarray(np.eye(3) * 19.2)
    args = (0, s["coordinates"], s["multipoles"], s["exclusions"], 0.5, 16, 4, 1, "THOLE", s["damping_factors"], True,
            box)
    monkeypatch.setenv("FMM_GB300_M2L_BYTES", "1000")
    P = fmm_gb300.field_fmm(*args)
    assert fmm_gb300.last_stats()["t_m2l_product"] <= 0.0
    O = oracle.field_fmm(*args)
    assert rel_err(P, O, slice(1, None)) <= 1e-12
    assert potential_up_to_constant(P, O)[0] <= 1e-12


def test_large_groups_are_not_limited(monkeypatch):
    """Exact coefficients, more than 16 pairs a group: the products, whatever the limit."""
    s = systems.water(2000, 49.0, seed=4)
    args = (0, s["coordinates"], s["multipoles"], s["exclusions"], 0.5, 32, 6, 1, "THOLE", s["damping_factors"])
    monkeypatch.setenv("FMM_GB300_M2L_BYTES", "1000")
    fmm_gb300.field_fmm(*args, options=Options.exact())
    s = fmm_gb300.last_stats()
    assert s["m2l_pairs"] > 16 * s["m2l_groups"] and s["t_m2l_product"] > 0.0


def test_plan(monkeypatch):
    """A plan keeps the choice made with its lists."""
    s = systems.water(400, 29.0, seed=9)
    monkeypatch.setenv("FMM_GB300_M2L_BYTES", "1000")
    plan = fmm_gb300.Plan(s["coordinates"], 10, s["exclusions"], 0.5, 32, 5, 1, "THOLE", s["damping_factors"])
    monkeypatch.delenv("FMM_GB300_M2L_BYTES")
    F = plan.execute(s["multipoles"])
    args = (0, s["coordinates"], s["multipoles"], s["exclusions"], 0.5, 32, 5, 1, "THOLE", s["damping_factors"])
    assert rel_err(F, oracle.field_fmm(*args)) <= 1e-12
