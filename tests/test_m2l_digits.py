"""CPU restatement of the FP64 M2L product's digit sums (csrc/m2l_tc64.cuh): FP32
accumulators of products of base-256 digits, with the digits that make them as
large as they can be.  Within a segment every weight to 256^-5 is exact, and what
256^-6 and 256^-7 round off is below an eighth of what the products left out
(weight 256^-8) can be: of the 7 x 176 additions at 256^-6 the last 37 are beyond
2^24, where one rounds by a unit at most."""
import os
import re

import numpy as np
import pytest

SRC = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fmm_gb300", "csrc",
                        "m2l_tc64.cuh")).read()


def constant(name):
    m = re.search(r"constexpr int %s = (\d+);" % name, SRC)
    assert m, name
    return int(m.group(1))


def accumulate(K, d, lead, rest):
    """Sum of K components' digit products of weight 256^-d, one FP32 addition
    each, and the exact one."""
    a = np.array([lead] + [rest] * 7, dtype=np.int64)
    prod = [int(a[i] * a[d - i]) for i in range(d + 1)]
    acc, exact = np.float32(0.0), 0
    for _ in range(K):
        for p in prod:
            acc = np.float32(acc + np.float32(p))
            exact += p
    return int(acc), exact


@pytest.mark.parametrize("lead,rest", [(64, 127), (-64, -128), (63, 85), (1, -127)])
@pytest.mark.parametrize("d", range(8))
def test_segment(d, lead, rest):
    K = constant("kD64Segment") * constant("kD64K")
    acc, exact = accumulate(K, d, lead, rest)
    left_out = 7 * K * 2 ** 14 / 256.0  # in units of 256^-7
    if d <= 5:
        assert acc == exact
    assert abs(acc - exact) * 256.0 ** (7 - d) <= left_out / 8.0


def test_whole_basis_is_too_long():
    """All Cartesian components of order 12 in one accumulator would round."""
    acc, exact = accumulate(455, 3, -64, -128)
    assert acc != exact or exact > 2 ** 24
    assert constant("kD64Segment") * constant("kD64K") * 5 <= 1024 < 455 * 3


def test_reduced_basis_is_one_segment():
    assert constant("kD64Segment") * constant("kD64K") >= 13 ** 2
