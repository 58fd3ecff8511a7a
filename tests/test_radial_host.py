"""CPU check of the FP32 radial functions (csrc/pair.cuh, compiled here as host
code): the ERF kernel's Boys table is indexed by a r^2, which factors of both
signs make negative and a NaN factor unordered.  Those give NaN, as the root of a
does, and read nothing before or behind the table: the code is compiled with
bounds checks on it.  In range, the values against FP64 ones."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fmm_gb300", "csrc")
SOURCE = """
#include <cmath>
static inline float rsqrtf(float x) { return 1.0f / std::sqrt(x); }
#include "pair.cuh"
template <int N> static void run(double r2, double a, float* g, double* h) {
    const float r2f = (float)r2;
    const double ir = 1.0 / std::sqrt((double)r2f);
    const float irf = (float)ir;
    fmm::radial_g_ir<N, float>(3, r2f, irf, (float)a, g, (float)(ir / irf - 1.0));
    fmm::radial_g_ir<N, double>(3, (double)r2f, ir, (double)(float)a, h, 0.0);
}
extern "C" void erf_g(int n, double r2, double a, float* g, double* h) {
    if (n == 1) run<1>(r2, a, g, h);
    else if (n == 2) run<2>(r2, a, g, h);
    else run<4>(r2, a, g, h);
}
"""
FLAGS = ["-std=c++17", "-O1", "-w", "-x", "c++", "-D__host__=", "-D__device__=", "-D__constant__=", "-D__forceinline__=inline",
         "-D__noinline__=", "-fsanitize=bounds-strict,float-cast-overflow", "-fsanitize-undefined-trap-on-error"]


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    """n r2 a on each line of stdin; g and h out."""
    d = tmp_path_factory.mktemp("radial")
    src, exe = d / "t.cpp", d / "t"
    src.write_text(SOURCE + """
#include <cstdio>
int main() {
    int n; double r2, a;
    while (std::scanf("%d %lf %lf", &n, &r2, &a) == 3) {
        float g[5] = {}; double h[5] = {};
        erf_g(n, r2, a, g, h);
        for (int j = 0; j <= n; ++j) std::printf("%.9g %.17g ", g[j], h[j]);
        std::printf("\\n");
        std::fflush(stdout);
    }
}
""")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.check_call(["g++"] + FLAGS + ["-I", CSRC, "-I", os.path.join(cuda, "include"), "-o", str(exe), str(src)])
    return str(exe)


def evaluate(program, rows):
    out = subprocess.run([program], input="".join("%d %.17g %.17g\n" % r for r in rows), capture_output=True, text=True)
    assert out.returncode == 0, "stopped at %r" % (rows[len(out.stdout.splitlines())],)
    v = [np.array(line.split(), dtype=float).reshape(-1, 2) for line in out.stdout.splitlines()]
    assert len(v) == len(rows)
    return v


@pytest.mark.parametrize("n", [1, 2, 4])
def test_out_of_range(program, n):
    rows = [(n, r2, a) for r2 in (1e-3, 1.0, 30.0, 1e4) for a in (-1e-3, -0.5, -1e3, -1e30, float("nan"))]
    for (g, row) in zip(evaluate(program, rows), rows):
        assert np.all(np.isnan(g[:, 0])), row


@pytest.mark.parametrize("n", [1, 2, 4])
def test_in_range(program, n):
    """Bar: 1e-6, some twenty FP32 roundings in the polynomial, the recursion and
    the powers."""
    s = np.concatenate([[0.0], np.geomspace(1e-6, 0.99, 20), np.arange(1.0, 40.0, 0.37), [23.9999, 24.0, 28.0, 31.999, 32.0]])
    rows = [(n, max(v, 1e-7) / 0.3 if v else 1e-6, 0.3 if v else 0.0) for v in s]
    rows = [r for r in rows if r[2] > 0.0]
    for (g, row) in zip(evaluate(program, rows), rows):
        assert np.all(np.abs(g[:, 0] - g[:, 1]) <= 1e-6 * np.abs(g[:, 1])), (row, g)


@pytest.mark.parametrize("n,bars", [(1, [9.5e-8, 1.22e-7]), (2, [9.4e-8, 1.16e-7, 1.20e-7]),
                                    (4, [9.3e-8, 1.15e-7, 1.15e-7, 1.38e-7, 1.33e-7])])
def test_accuracy(program, n, bars):
    """rms errors: the bars are those of the plain series and error function."""
    rng = np.random.default_rng(0)
    s = np.exp(rng.uniform(np.log(1e-3), np.log(40.0), 6000))
    a = rng.uniform(0.09, 0.64, 6000)
    v = np.array(evaluate(program, [(n, x / b, b) for x, b in zip(s, a)]))
    rms = np.sqrt(np.mean((v[:, :, 0] / v[:, :, 1] - 1.0) ** 2, axis=0))
    assert np.all(rms <= bars), rms
