"""The sequential root centre (csrc/tree.cu seq_sum) where its sum changes
binade all the time: coordinates around zero.  One FP64 addition after the other,
200,000 particles take 7.4 ms; a parallel form with a block's attempt at each
change took 8.5 to 12.5 ms, with a tree of 0.7 ms where the sum grows steadily; the
whole tree is to stay below ten times that.  And the bits of the result there:
ties, sums that nowhere round."""
import numpy as np
import pytest
import torch

import fmm_gb300
from fmm_gb300 import Options

pytestmark = pytest.mark.gpu

N = 199998


def _tree_time(X):
    n = len(X)
    put = lambda a: torch.from_numpy(np.ascontiguousarray(a.T)).cuda().t()  # noqa: E731
    M = np.random.default_rng(1).normal(size=(n, 1))
    dev = put(X), put(M), put(np.arange(1, n + 1, dtype=np.int32)[:, None])
    F = torch.zeros((1, n), dtype=torch.float64, device="cuda").t()
    times = []
    for _ in range(4):
        fmm_gb300.field_fmm_device(*dev, 0.9, 512, 2, 0, F, options=Options())
        times.append(fmm_gb300.last_stats()["t_tree"])
    return min(times)


@pytest.mark.parametrize("kind", ["centred", "gauss", "lattice"])
def test_tree_time(kind):
    rng = np.random.default_rng(4)
    if kind == "lattice":
        g = 2.5 * np.arange(-29, 30)
        X = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)[:N]
    else:
        X = {"centred": lambda: rng.uniform(-73.0, 73.0, (N, 3)), "gauss": lambda: 40.0 * rng.normal(size=(N, 3))}[kind]()
    assert _tree_time(X) < 10.0 * _tree_time(rng.uniform(0.0, 146.0, (N, 3)))


def _values(kind, n, rng):
    if kind == "lattice":
        return 2.5 * (np.arange(n) % 59 - 29)
    if kind == "float32":
        return rng.uniform(-73.0, 73.0, n).astype(np.float32).astype(np.float64)
    if kind == "ties":  # sums of 2^20 in which a third of the terms are half a unit
        return np.concatenate([[2.0 ** 20], np.ldexp(rng.integers(-9, 10, n - 1) / 2.0, -32)])
    if kind == "negative_ties":
        return np.concatenate([[-2.0 ** 20], np.ldexp(rng.integers(-9, 10, n - 1) / 2.0, -32)])
    # units of 2^-40 until the sum needs more bits than 53
    return np.ldexp(rng.integers(0, 1 << 44, n).astype(np.float64), -40)


@pytest.mark.parametrize("n", [65, 129, 4096, 4097, 30011])
@pytest.mark.parametrize("kind", ["lattice", "float32", "ties", "negative_ties", "exact_then_not"])
def test_bits(kind, n):
    """Host calls add one term after the other: the same trees and fields."""
    rng = np.random.default_rng(n)
    X = np.stack([_values(kind, n, rng), rng.uniform(-30.0, 30.0, n), _values("float32", n, rng)], axis=1)
    X = np.asfortranarray(X)
    M = np.asfortranarray(rng.normal(size=(n, 1)))
    E = np.arange(1, n + 1, dtype=np.int32)[:, None]
    put = lambda a: torch.from_numpy(np.ascontiguousarray(a.T)).cuda().t()  # noqa: E731
    F = torch.zeros((1, n), dtype=torch.float64, device="cuda").t()
    opt = Options(coef_mode="exact", excl_mode="mask")
    fmm_gb300.field_fmm_device(put(X), put(M), put(E), 0.5, 64, 4, 0, F, options=opt)
    torch.cuda.synchronize()
    assert np.array_equal(F.cpu().numpy(), fmm_gb300.field_fmm(0, X, M, E, 0.5, 64, 4, 0, options=opt))
