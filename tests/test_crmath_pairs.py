"""The double-float exp / log / pow and product differences of the GPU samplers
(xitils_gb300/csrc/crmath.cuh), compiled for the host and compared with the
double-precision expressions whose rounding they reproduce.

exp, log and pow keep a result only when its rounding is certain within their error bound
and otherwise call the double-precision function, so they differ from it only where the
double result itself was rounded across a float boundary (2^-29 per call). The product
differences and the multiples of pi round an exact sum of floats once, against the
double's two roundings: about 2^-26 per call. Over a million arguments each, at most
one difference is allowed.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r'''
#include "crmath.cuh"
#include <cmath>
using namespace xgb;
extern "C" void cr_eval(int what, int n, const float* a, const float* b, const float* c, const float* d, float* o, float* r) {
    const double pi = 3.14159265358979323846;
    for (int i = 0; i < n; ++i) {
        switch (what) {
        case 0: o[i] = crExpf(a[i]); r[i] = (float)exp((double)a[i]); break;
        case 1: o[i] = crLogf(a[i]); r[i] = (float)log((double)a[i]); break;
        case 2: o[i] = crPowf(a[i], b[i]); r[i] = (float)pow((double)a[i], (double)b[i]); break;
        case 3: o[i] = cr::diffProd(a[i], b[i], c[i], d[i]); r[i] = (float)((double)a[i] * b[i] - (double)c[i] * d[i]); break;
        case 4: o[i] = crTwoPi(a[i]); r[i] = (float)(2.0 * pi * (double)a[i]); break;
        case 5: o[i] = crMinusPi(a[i]); r[i] = (float)((double)a[i] - pi); break;
        case 6: o[i] = crOverPi(a[i]); r[i] = (float)((double)a[i] / pi); break;
        case 7: o[i] = crCubef(a[i]); r[i] = (float)pow((double)a[i], 3.0); break;
        }
    }
}
'''
N = 1_000_000


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    inc = next((os.path.join(p, "include") for p in (os.environ.get("CUDA_HOME"), "/usr/local/cuda")
                if p and os.path.exists(os.path.join(p, "include", "cuda_runtime.h"))), None)
    if inc is None:
        pytest.skip("cuda_runtime.h not found")
    d = tmp_path_factory.mktemp("crpairs")
    (d / "cr.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off", "-w",
                    "-I", os.path.join(ROOT, "xitils_gb300", "csrc"), "-I", inc, str(d / "cr.cpp"), "-o",
                    str(d / "libcr.so")], check=True, capture_output=True)
    return C.CDLL(str(d / "libcr.so"))


def _differ(lib, what, *args):
    a = [np.ascontiguousarray(x, dtype=np.float32) for x in args]
    a += [a[0]] * (4 - len(a))
    o, r = np.empty_like(a[0]), np.empty_like(a[0])
    fp = lambda x: x.ctypes.data_as(C.POINTER(C.c_float))
    lib.cr_eval(what, a[0].size, *[fp(x) for x in a], fp(o), fp(r))
    return int(np.sum((o != r) & ~(np.isnan(o) & np.isnan(r))))


def _cases(what):
    rng = np.random.default_rng(what)
    u = lambda: rng.random(N)
    if what == 0:  # kappa (cos - 1) and -2 kappa: past the underflow, the subnormal band, tiny arguments
        return [np.concatenate([-u() * np.exp(u() * 12 - 5), [0.0, -0.0, -87.0, -87.01, -103.9, -104.0, -104.01, -1e30,
                                                             -np.inf, np.nan, 88.0, 89.0, np.inf, 1e-30]])]
    if what == 1:
        return [np.concatenate([u(), 1.0 - 1e-3 * u(), [1.0, 0.0, -1.0, 2.0, 1.9999999, 1e-40, 1e30, np.inf, np.nan]])]
    if what == 2:  # x ^ (2 / (s + 1)) and x ^ (1 / (s + 1)) for sharpness s
        y = np.where(u() < 0.5, 1.0, 2.0) / (np.exp(12 * u() - 3) + 1.0)
        sx = np.array([0.0, 1.0, 0.5, 2.0, -0.5, 2.0 ** -41, 0.0, 0.3, 0.3, np.nan, 0.5], np.float64)
        sy = np.array([0.5, 0.5, 2.0, 0.5, 0.5, 0.5, -1.0, 0.0, np.inf, 0.5, np.nan], np.float64)
        return [np.concatenate([u(), sx]), np.concatenate([y, sy])]
    if what == 3:  # generic, nearly parallel (cancelling), components of very different size, zeros
        v = [2 * u() - 1 for _ in range(4)]
        k = N // 4
        v[2][:k], v[3][:k] = v[0][:k] * (1 + 1e-6 * (u()[:k] - 0.5)), v[1][:k]
        v[1][k:2 * k] *= np.exp(-20 * u()[:k])
        v[3][2 * k:3 * k] = 0.0
        return v
    if what == 4:
        return [(rng.integers(0, 1 << 32, N).astype(np.float32) * np.float32(2.0 ** -32))]
    if what == 5:
        return [np.float32(2 * np.pi) * rng.random(N, dtype=np.float32)]
    return [np.concatenate([u(), [0.0, 1.0]])]


@pytest.mark.parametrize("what", range(8))
def test_rounds_as_the_double_expression(lib, what):
    assert _differ(lib, what, *_cases(what)) <= 1
