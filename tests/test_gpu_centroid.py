"""The root centre of device calls (csrc/tree.cu seq_sum) is the sequential sum
of the host's, bit for bit: the trees, and with them the fields, of the device
and the host entry are the same."""
import numpy as np
import pytest
import torch

import fmm_gb300
from fmm_gb300 import Options
from test_gpu_parity import _gpu_tree

pytestmark = pytest.mark.gpu


def _values(kind, n, rng):
    if kind == "box":
        return 158.0 * rng.random(n)
    if kind == "centred":
        return 50.0 * (rng.random(n) - 0.5)
    if kind == "eighths":  # many ties
        return np.floor(400.0 * rng.random(n)) / 8.0
    if kind == "alternating":
        return np.where(np.arange(n) % 2, -1.0, 1.0) * (20.0 + 1e-9 * rng.random(n))
    if kind == "scales":
        return np.ldexp(rng.random(n) - 0.5, rng.integers(-40, 6, n))
    if kind == "offset":
        return -1.0e6 - 30.0 * rng.random(n)
    return np.where(np.arange(n) < n // 2, 0.0, rng.random(n) * 30.0)  # zeros first


KINDS = ["box", "centred", "eighths", "alternating", "scales", "offset", "zeros"]


@pytest.mark.parametrize("n", [100, 1023, 4097, 20011])
@pytest.mark.parametrize("k", range(len(KINDS)))
@pytest.mark.parametrize("centroid", ["sequential", "blocked"])
def test_device_centroid(n, k, centroid):
    rng = np.random.default_rng(n + k)
    X = np.asfortranarray(np.stack([_values(KINDS[(k + d) % len(KINDS)], n, rng) for d in (0, 2, 5)], axis=1))
    M = np.asfortranarray(rng.normal(size=(n, 1)))
    E = np.asfortranarray(np.arange(1, n + 1, dtype=np.int32)[:, None])
    opt = Options(coef_mode="exact", excl_mode="mask", centroid_mode=centroid)
    dev = [torch.from_numpy(np.ascontiguousarray(a.T)).cuda().t() for a in (X, M, E)]  # column-major
    F = torch.zeros((1, n), dtype=torch.float64, device="cuda").t()
    if centroid == "sequential":
        fmm_gb300.field_fmm_device(dev[0], dev[1], dev[2], 0.5, 64, 4, 0, F, options=opt)
        torch.cuda.synchronize()
        H = fmm_gb300.field_fmm(0, X, M, E, 0.5, 64, 4, 0, options=opt)
        assert np.array_equal(F.cpu().numpy(), H)
    else:  # 1,024 lanes added on the device, then their sums in order
        c = [sum_in_order([sum_in_order(X[i::1024, d]) for i in range(1024)]) / n for d in range(3)]
        assert np.array_equal(_gpu_tree(X, 64, 0.5, 1)["center"][0], c)


def sum_in_order(v):
    s = 0.0
    for x in v:
        s += float(x)
    return s
