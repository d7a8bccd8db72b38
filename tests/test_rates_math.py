"""The rate kernels' exponential, logarithm, reciprocal and quotient (csrc/rates_math.cuh) against 80-bit
references, compiled for the host: the functions are plain FMAs, table reads and integer arithmetic but for the
hardware's approximate reciprocal, which is stood in for by the exact one cut to the documented 20 bits."""
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tiger_nga_b200", "csrc")

STUB = r"""
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#define __device__
#define __constant__
#define __forceinline__ inline
struct double2 { double x, y; };
struct Idx { int x; };
static const Idx threadIdx{0}, blockDim{1};
inline void __syncthreads() {}
using std::fma;
using std::min;
inline uint64_t bits(double x) { uint64_t u; std::memcpy(&u, &x, 8); return u; }
inline double from_bits(uint64_t u) { double x; std::memcpy(&x, &u, 8); return x; }
inline int __double2loint(double x) { return (int)(uint32_t)bits(x); }
inline int __double2hiint(double x) { return (int)(uint32_t)(bits(x) >> 32); }
inline double __hiloint2double(int h, int l) { return from_bits((uint64_t)(uint32_t)h << 32 | (uint32_t)l); }
inline double __longlong_as_double(long long u) { return from_bits((uint64_t)u); }
inline double approx_rcp(double b) {  // truncated: an error up to 2^-20, the result flushed like the operand
  const double r = std::fabs(b) > 0x1p1022 ? 0.0 : from_bits(bits(1.0 / b) & ~((1ull << 32) - 1));
  return r;
}
#define asm(...) r = approx_rcp(b)
"""

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "rates_math.cuh"
using namespace tng;
int main(int argc, char** argv) {  // op, then pairs of doubles on stdin: value and error in units of the last place
  alignas(16) static double xt[kMathTab];
  stage_math_tab(xt);
  double in[2];
  while (std::fread(in, 8, 2, stdin) == 2) {
    const double x = in[0], b = in[1];
    double v = 0.0;
    long double ref = 0.0L;
    switch (argv[1][0]) {
      case 'e': v = tng_exp(x, xt), ref = expl((long double)x); break;
      case 's': v = tng_exp<true>(x, xt), ref = expl((long double)x); break;
      case 'l': v = tng_log(x, xt), ref = logl((long double)x); break;
      case 'r': v = tng_rcp(x), ref = 1.0L / x; break;
      case 'q': v = tng_quot(x, b), ref = (long double)x / b; break;
    }
    int e;
    std::frexp((double)ref, &e);
    const double out[3] = {v, (double)((v - ref) / ldexpl(1.0L, e - 53)), (double)(v - ref)};
    std::fwrite(out, 8, 3, stdout);
  }
}
"""


@pytest.fixture(scope="module")
def math(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("rates_math")
    (d / "cuda_runtime.h").write_text(STUB)
    (d / "m.cpp").write_text(PROGRAM)
    subprocess.check_call([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", str(d), "-I", CSRC, str(d / "m.cpp"),
                           "-o", str(d / "m")])

    def call(op, x, b=None):
        """Values, errors in units of the last place of the exact result, absolute errors."""
        a = np.stack([x, np.zeros_like(x) if b is None else b], axis=1)
        r = subprocess.run([str(d / "m"), op], input=a.tobytes(), stdout=subprocess.PIPE, check=True)
        return np.frombuffer(r.stdout).reshape(-1, 3).T

    return call


G = np.random.default_rng(3)


def near(points, n=40):
    """Neighbours of the points, on both sides."""
    p = np.repeat(np.asarray(points, dtype=np.float64), 2 * n + 1)
    return p + np.tile(np.arange(-n, n + 1), len(points)) * np.spacing(p)


def test_exponential(math):
    ln2 = np.log(2.0)
    x = np.concatenate([G.uniform(-40, 40, 400_000), G.uniform(-708, 709, 400_000), G.uniform(-1, 1, 100_000) * 2.0 ** -20,
                        near((np.arange(-300, 300) + 0.5) * ln2 / 256)])
    v, ulp, _ = math("e", x)
    assert np.abs(ulp).max() <= 1.4
    assert np.mean(np.abs(ulp) > 1.0) <= 0.005
    v, ulp, _ = math("s", -np.minimum(np.abs(x), 708.0))  # the saturating form
    assert np.abs(ulp).max() <= 1.4


def test_exponential_outside_its_range(math):
    x = np.concatenate([[-4.9e6, -1e5, -746.0], G.uniform(-4.9e6, -746.0, 10_000)])
    assert np.all(np.abs(math("e", x)[0]) <= 2.3e-308)
    assert np.all(np.abs(math("s", x)[0]) <= 2.3e-308)
    x = np.concatenate([[710.0, 1e5, 4.9e6], G.uniform(710.0, 4.9e6, 10_000)])
    assert not np.isfinite(math("e", x)[0]).any()
    v = math("s", x)[0]
    assert np.isfinite(v).all() and (v >= 2.0 ** 1023).all()
    assert np.isnan(math("e", np.array([np.nan]))[0]).all() and np.isnan(math("s", np.array([np.nan]))[0]).all()


def test_logarithm(math):
    x = np.concatenate([10.0 ** G.uniform(-300, 300, 400_000), G.uniform(0.5, 2.0, 400_000), 1.0 + G.uniform(-1, 1, 100_000) * 1e-6,
                        near(1.0 + (np.arange(128) + 0.5) / 128), near([1.0, 2.0, 0.5, 1e-300])])
    v, ulp, err = math("l", x)
    # the absolute error is bounded near one, where ln x vanishes, the relative one elsewhere
    close = np.abs(np.log(x)) < 0.4
    assert np.abs(ulp[~close]).max() <= 2.0
    assert np.abs(err[close]).max() <= 1e-16
    assert np.abs(ulp[close & (x > 1.0) & (x < 1.4)]).max() <= 5.5
    assert math("l", np.array([1.0]))[0][0] == 0.0
    assert np.isnan(math("l", np.array([-1.0, np.inf, np.nan, -0.0]))[0]).all()
    v = math("l", np.array([0.0, 5e-324, 1e-310, 2.2e-308]))[0]  # below the normal range
    assert np.all((v >= -709.1) & (v <= -708.3))


def test_reciprocal_and_quotient(math):
    b = np.concatenate([1.0 + 10.0 ** G.uniform(-18, 300, 400_000), G.uniform(1.0, 2.0, 400_000)])
    v, ulp, _ = math("r", b)
    assert np.abs(ulp).max() <= 0.51
    assert np.all(math("r", np.array([2.0 ** 1023, 1.7e308]))[0] == 0.0)
    a = G.choice([-1.0, 1.0], b.size) * 10.0 ** G.uniform(-5, 6, b.size)
    d = 10.0 ** G.uniform(-8, 12, b.size)
    v, ulp, _ = math("q", a, d)
    assert np.abs(ulp).max() <= 0.51  # one correction by the FMA residual: rounded correctly but near a tie
