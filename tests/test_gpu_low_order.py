"""Expansion orders below the multipole order: the source moments above the
expansion order reach no output (csrc/translate.cu k_p2m)."""
import numpy as np
import pytest

import fmm_gb300
import oracle
from fmm_gb300 import Options, systems
from helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,p", [(1, 0), (2, 0), (2, 1), (3, 2)])
def test_order_below_multipoles(m, p):
    s = systems.water(700, 35.0, order=m, seed=p)
    args = (0, s["coordinates"], s["multipoles"], s["exclusions"], 0.5, 32, p, 1)
    kw = dict(coef_mode="exact", excl_mode="mask")
    G = fmm_gb300.field_fmm(*args, options=Options(**kw))
    O = oracle.field_fmm(*args, **kw)
    assert np.all(np.isfinite(G))
    assert rel_err(G, O) <= 1e-12
