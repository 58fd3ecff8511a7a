"""FP64 M2L products over all Cartesian components in several accumulation
segments (csrc/m2l_tc64.cuh kD64Segment: 176 components; 220, 286, 364 and 455
at orders 9 to 12) against the CPU oracle.  Bar: the FP64 path's, 1e-12."""
import pytest

import fmm_gb300
import oracle
from fmm_gb300 import systems
from helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [8, 9, 11, 12])
@pytest.mark.parametrize("n_mol,ncrit", [(150, 16), (600, 24)])
def test_reference_tensors(p, n_mol, ncrit):
    s = systems.water(n_mol, (59.05 * n_mol) ** (1 / 3), seed=p)
    args = (0, s["coordinates"], s["multipoles"], s["exclusions"], 0.6, ncrit, p, 1, "THOLE", s["damping_factors"])
    G = fmm_gb300.field_fmm(*args)
    assert fmm_gb300.last_stats()["t_m2l_product"] > 0.0
    assert rel_err(G, oracle.field_fmm(*args)) <= 1e-12
