"""The double-float reciprocal of the projector's pivots (DF64::rrecip), compiled
for the host with the rounding intrinsics of the same names: over mantissas
and exponents it must be as accurate as a binary64 quotient split into two
floats.  Bound: the split's own rounding, half a unit of the low word, which is
at most 2^-24 of the high word's binade -- 2^-49 relative -- and 2^-60 on top
for the sums before it."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "qutree_gb300", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

SHIM = r"""
#include <cmath>
#include <cuda_runtime.h>
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
inline float __frcp_rn(float a) { return 1.0f / a; }
inline float __double2float_rn(double a) { return (float)a; }
template <class T> inline T __ldg(const T* p) { return *p; }
using std::fma;
#include "qt_arith.cuh"
extern "C" void rrecip(const float* hi, const float* lo, float* rh, float* rl, int n) {
  for (int i = 0; i < n; ++i) {
    const float2 r = qt::DF64::rrecip(make_float4(hi[i], lo[i], 0.f, 0.f));
    rh[i] = r.x;
    rl[i] = r.y;
  }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    d = tmp_path_factory.mktemp("df")
    src, so = str(d / "df.cpp"), str(d / "df.so")
    with open(src, "w") as f:
        f.write(SHIM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC,
                    "-I", os.path.join(CUDA, "include"), src, "-o", so], check=True)
    return ctypes.CDLL(so)


@pytest.mark.parametrize("exponent", [-60, -1, 0, 1, 40])
def test_reciprocal_has_the_split_quotients_accuracy(lib, exponent):
    rng = np.random.default_rng(abs(exponent))
    x = np.concatenate([1.0 + rng.random(100000), 1.0 + 2.0 ** -rng.integers(1, 48, 1000),
                        2.0 - 2.0 ** -rng.integers(1, 48, 1000)]) * 2.0 ** exponent
    hi = x.astype(np.float32)
    lo = (x - hi.astype(np.float64)).astype(np.float32)
    rh, rl = np.empty_like(hi), np.empty_like(hi)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    lib.rrecip(p(hi), p(lo), p(rh), p(rl), len(hi))
    # 1 - x r in exact integer arithmetic
    worst = 0.0
    for h, l, a, b in zip(hi.tolist(), lo.tolist(), rh.tolist(), rl.tolist()):
        s = 1 << 200
        xi, ri = int(h * 2.0 ** 120) + int(l * 2.0 ** 120), int(a * 2.0 ** 150) + int(b * 2.0 ** 150)
        d = xi * ri - (1 << 270)
        worst = max(worst, abs(d) / s / 2.0 ** 70)
    assert worst <= 2.0 ** -49 + 2.0 ** -60
