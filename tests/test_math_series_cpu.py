"""The series of gft_math.cuh, compiled for the host, against 80-bit long doubles (no GPU).

The header's device functions are plain C++ but for a few bit casts, so g++ compiles them as they are,
with hardware fused multiply-adds and no contraction of its own.  Bars: the rounding of the last
operation, 2^-24 or 2^-53 of the result, and what the comments of the header state beside it.
"""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gftevolver_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#define __device__
#define __noinline__
#define __forceinline__ inline
template <class To, class From> static To cast(From f) { To t; std::memcpy(&t, &f, sizeof t); return t; }
static unsigned __float_as_uint(float f) { return cast<unsigned>(f); }
static float __uint_as_float(unsigned u) { return cast<float>(u); }
static long long __double_as_longlong(double d) { return cast<long long>(d); }
static double __longlong_as_double(long long l) { return cast<double>(l); }
static int __double2hiint(double d) { return (int)(cast<unsigned long long>(d) >> 32); }
static unsigned max(unsigned a, unsigned b) { return a > b ? a : b; }
#define __CUDA_RUNTIME_H__  // the header's own include brings nothing more
#include "gft_math.cuh"

typedef long double Long;
static Long long_sqrt1m(Long c) { return -c / (1 + sqrtl(1 - c)); }
static Long long_sin(Long x) { return sinl(x); }
static Long long_cos(Long x) { return cosl(x); }
static Long long_asin(Long x) { return asinl(x); }

// The largest error of f(x) over 2 million x, logarithmically spread over [lo, hi], as T.
template <class T, class F>
static void report(const char* name, double lo, double hi, bool relative, F f, Long (*exact)(Long))
{
    std::mt19937_64 rng(7);
    std::uniform_real_distribution<double> u(std::log(lo), std::log(hi));
    double worst = 0;
    for (int i = 0; i < 2000000; i++) {
        const T x = (T)std::exp(u(rng));
        const Long e = exact(x);
        Long d = fabsl((Long)f(x) - e);
        if (relative) d /= fabsl(e);
        worst = std::fmax(worst, (double)d);
    }
    std::printf("%s %.6e\n", name, worst);
}

int main()
{
    using namespace gft;
    report<float>("sqrt1m_float", 1e-12, 1.0 / 64, true, [](float c) { return sqrt1m_series(c); }, long_sqrt1m);
    report<double>("sqrt1m_double", 1e-12, 1.0 / 64, true, [](double c) { return sqrt1m_series(c); }, long_sqrt1m);
    report<double>("sin_double", 1e-9, 1.5707963267948966, true, [](double r) { return sin_poly(r); }, long_sin);
    auto cosine = [](double r) { double s, c; sincos_poly(r, s, c); return c; };
    report<double>("cos_double", 1e-9, 1.5707963267948966, false, cosine, long_cos);
    report<double>("cos_double_small", 1e-9, 0.3, false, cosine, long_cos);
    report<float>("asin_float", 1e-6, 0.25, true, [](float x) { return asin_series(x); }, long_asin);
    report<double>("asin_double", 1e-9, 0.125, true, [](double x) { return asin_series(x); }, long_asin);
}
"""


@pytest.fixture(scope="module")
def errors(tmp_path_factory):
    cxx = os.environ.get("CXX", "g++")
    if not shutil.which(cxx):
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("series")
    (d / "series.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-O2", "-std=c++17", "-mfma", "-ffp-contract=off", "-I", CSRC, "-I",
                    os.path.join(CUDA, "include"), "-o", str(d / "series"), str(d / "series.cpp")],
                   check=True)
    out = subprocess.run([str(d / "series")], check=True, stdout=subprocess.PIPE, text=True).stdout
    return {k: float(v) for k, v in (line.split() for line in out.splitlines())}


def test_sqrt1m_rounds_once(errors):
    """-c/2 + c^2 G(c): one rounding, a few more of a term below 1/256 of it, and the fit's error."""
    assert errors["sqrt1m_float"] <= 2.0 ** -24 * (1 + 4 / 256) + 1.2e-8
    assert errors["sqrt1m_double"] <= 2.0 ** -53 * (1 + 6 / 256) + 8.4e-19


def test_sines_and_arcsines_round_once_or_twice(errors):
    """x + x^3 P(x^2): one rounding of the sum, and three of a term below x / 6 (asin) or 0.58 x (sin)."""
    assert errors["asin_float"] <= 2.0 ** -24 * (1 + 4 / 96)
    assert errors["asin_double"] <= 2.0 ** -53 * (1 + 4 / 384) + 4.5e-19
    assert errors["sin_double"] <= 2.0 ** -53 * (1 + 3 * 0.58) + 2.8e-19


def test_cosine_of_a_small_angle_keeps_its_half(errors):
    """1 + r^2 Q(r^2), |r| <= 0.3: half an ulp of the sum, of r^2 (below 2^-3) times 1/2, and of Q (below
    1/2) times r^2; nothing of the leading coefficient."""
    assert errors["cos_double_small"] <= 2.0 ** -54 + 0.5 * 2.0 ** -57 + 0.09 * 2.0 ** -55 + 1e-19
    assert errors["cos_double"] <= 2.0 ** -53 * (0.5 + 1 + 1.24)
