"""The pair arithmetic of the speckle post-processing (nmc_gb300/csrc/speckle_math.cuh), compiled for the host without
contraction: each function is within 0.51 units in the last place of its exact value, which is a double function's result
rounded once plus 2^-31 of the value."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include <cmath>
#include <cstring>
#define __device__
#define __forceinline__ inline
#define __noinline__
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
static inline float __fsqrt_rn(float a) { return std::sqrt(a); }
static inline float __fdividef(float a, float b) { return a / b; }
static inline float __int_as_float(int i) { float f; std::memcpy(&f, &i, 4); return f; }
using std::fabs;
#include "speckle_math.cuh"
extern "C" {
void v_sin(const float* x, float* y, int n) { for (int i = 0; i < n; ++i) y[i] = nmc::sin_ref(x[i]); }
void v_exp(const float* x, float* y, int n) { for (int i = 0; i < n; ++i) y[i] = nmc::exp_ref(x[i]); }
void v_wrap(const float* x, float* y, int n) { for (int i = 0; i < n; ++i) y[i] = nmc::wrap_ref(x[i]); }
void v_interfere(const float* a, const float* c, const float* f, const float* e, float* y, int n) {
  for (int i = 0; i < n; ++i) y[i] = nmc::interfere(a[i], c[i], f[i], e[i]);
}
}
"""


@pytest.fixture(scope="session")
def math_lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("pairs")
    (d / "pairs.cpp").write_text(SRC)
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "nmc_gb300", "csrc"),
                    str(d / "pairs.cpp"), "-o", str(d / "pairs.so")], check=True)
    return C.CDLL(str(d / "pairs.so"))


def _call(f, *x):
    y = np.empty_like(x[0])
    f(*(C.c_void_p(q.ctypes.data) for q in x), C.c_void_p(y.ctypes.data), C.c_int(y.size))
    return y


def _ulps(got, exact):
    """|got - exact| in units of the last place of a float of `exact`'s size."""
    unit = np.exp2(np.maximum(np.floor(np.log2(np.maximum(np.abs(exact), 1e-45))), -126.0) - 23.0)
    return np.abs(got.astype(np.float64) - exact) / unit


def _near(points, k=200):
    """`points` and the k floats on each side of each."""
    p = np.asarray(points, np.float32).view(np.int32)[:, None] + np.arange(-k, k + 1, dtype=np.int32)[None, :]
    return p.reshape(-1).view(np.float32)


def test_sin(math_lib):
    r = np.random.default_rng(1)
    x = np.concatenate([r.uniform(-3.1416, 3.1416, 1_000_000), np.exp(r.uniform(-60, 1.1, 200_000)) * r.choice([-1, 1], 200_000)]).astype(np.float32)
    x = np.concatenate([x, _near(np.arange(1, 5) * np.pi / 4), _near([np.pi]), -_near(np.arange(1, 5) * np.pi / 4), np.zeros(1, np.float32)])
    assert _ulps(_call(math_lib.v_sin, x), np.sin(x.astype(np.float64))).max() <= 0.51


def test_exp(math_lib):
    r = np.random.default_rng(2)
    x = np.concatenate([r.uniform(-87.0, 0.0, 1_000_000), r.uniform(-1.0, 0.0, 500_000), -np.exp(r.uniform(-60, 0, 100_000))]).astype(np.float32)
    x = np.concatenate([x, -_near((np.arange(1, 120) - 0.5) * np.log(2.0)), np.zeros(1, np.float32)])
    x = x[x > -87.0]
    assert _ulps(_call(math_lib.v_exp, x), np.exp(x.astype(np.float64))).max() <= 0.51


def test_wrap(math_lib):
    r = np.random.default_rng(3)
    x = np.concatenate([r.uniform(-20.0, 20.0, 500_000), r.uniform(-4096.0, 4096.0, 500_000)]).astype(np.float32)
    x = np.concatenate([x, _near(np.arange(1, 600) * np.pi, 20), -_near(np.arange(1, 600) * np.pi, 20)])
    d = x.astype(np.float64)
    assert _ulps(_call(math_lib.v_wrap, x), np.arctan2(np.sin(d), np.cos(d))).max() <= 0.51


def test_interfere(math_lib):
    # the sum cancels where a = c and the beat is -1: what the pairs lose is 2^-44 of a + c
    r = np.random.default_rng(4)
    n = 500_000
    a, c = (np.exp(r.uniform(-60, 0, n)).astype(np.float32) for _ in range(2))
    c[: n // 2] = (a[: n // 2] * r.uniform(0.5, 2.0, n // 2)).astype(np.float32)
    c[: n // 8] = a[: n // 8]
    a[-10:] = 0.0
    f, e = r.uniform(-1, 1, n).astype(np.float32), np.exp(-r.exponential(1.0, n)).astype(np.float32)
    f[::5], e[::3] = -1.0, 1.0
    got = _call(math_lib.v_interfere, a, c, f, e)
    with np.errstate(under="ignore"):
        s, p = (a + c).astype(np.float64), (a * c).astype(np.float64)
    exact = (s + 2.0 * np.sqrt(p) * (f.astype(np.float64) * e.astype(np.float64))) / 4.0
    unit = np.exp2(np.maximum(np.floor(np.log2(np.maximum(np.abs(exact), 1e-45))), -126.0) - 23.0)
    assert np.all(np.abs(got - exact) <= 0.51 * unit + 2.0 ** -44 * s)
