"""The reciprocals, roots, quotients and powers of csrc/series.cuh, as the kernels
take them, on the CPU against wider arithmetic.  The estimates are FP32
numbers up to 2 ulp off (the instructions' stated error).  Bound: half an ulp for the
last rounding, the series' first dropped term ((2.4e-7)^3 and 5/16 of it,
below 1e-4 ulp) and the roundings of a correction of 2e-7 of the result (below
1e-6 ulp): 0.501 ulp; the short form of the root lets half of the rounding of s = x y
in as well, half an ulp of s: 0.751 ulp of the root, which shares s's binade, and
1.001 of its reciprocal, whose ulp may be half as large relative to it."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sph-dem_gb300", "csrc")

HARNESS = r"""
#include <algorithm>
#include <cfloat>
#include <cstdio>
#include <random>
#include "series.cuh"

/* |got - want| in units of the last place of want */
static double ulps(double got, long double want) {
    const double w = (double)want;
    return (double)(fabsl((long double)got - want) / (std::nextafter(fabs(w), INFINITY) - fabs(w)));
}
static float off(float x, int n) {
    for (; n > 0; n--) x = std::nextafterf(x, INFINITY);
    for (; n < 0; n++) x = std::nextafterf(x, 0.f);
    return x;
}

int main() {
    std::mt19937_64 rng(7);
    std::uniform_real_distribution<double> ex(-29.0, 29.0);
    double worst[5] = {0, 0, 0, 0, 0};
    for (int k = 0; k < 400000; k++) {
        const double x = std::pow(10.0, ex(rng));
        const int n = (int)(rng() % 5) - 2;
        const float yr = off((float)(1.0 / x), n), ys = off((float)(1.0 / std::sqrt(x)), n);
        worst[0] = std::max(worst[0], ulps(sphdem::rcp_series(x, yr), 1.0L / (long double)x));
        double inv = 0.0;
        const long double root = sqrtl((long double)x);
        worst[1] = std::max(worst[1], ulps(sphdem::sqrt_series_full(x, ys, &inv), root));
        worst[2] = std::max(worst[2], ulps(inv, 1.0L / root));
        worst[3] = std::max(worst[3], ulps(sphdem::sqrt_series(x, ys, &inv), root));
        worst[4] = std::max(worst[4], ulps(inv, 1.0L / root));
    }
    /* FP32 quotients: wider arithmetic is double */
    double q = 0.0;
    std::uniform_real_distribution<float> e2(-15.f, 15.f);
    for (int k = 0; k < 400000; k++) {
        const float a = std::pow(10.f, e2(rng)), b = std::pow(10.f, e2(rng));
        const float y = off((float)(1.0 / (double)b), (int)(rng() % 3) - 1);
        const double want = (double)a / (double)b;
        const float w = (float)want;
        q = std::max(q, fabs((double)sphdem::quotient(a, b, y) - want) / (double)(std::nextafterf(w, INFINITY) - w));
    }
    /* the gradient factor -10 C x^N of an FP32 x */
    double pw = 0.0;
    std::uniform_real_distribution<float> e3(-5.f, 5.f);
    for (int k = 0; k < 400000; k++) {
        const float x = std::pow(10.f, e3(rng));
        for (int n = 3; n <= 5; n++) {
            const double c = -10.0 * (n == 4 ? 7.0 / (64.0 * 3.14159265) : 21.0 / (256.0 * 3.14159265));
            const float g = (float)c, glo = (float)(c - (double)g);
            const float got = n == 3 ? sphdem::scaled_power<3>(x, g, glo)
                                     : (n == 4 ? sphdem::scaled_power<4>(x, g, glo) : sphdem::scaled_power<5>(x, g, glo));
            double want = c;
            for (int i = 0; i < n; i++) want *= (double)x;
            const float w = fabsf((float)want);
            pw = std::max(pw, fabs((double)got - want) / (double)(std::nextafterf(w, INFINITY) - w));
        }
    }
    for (double w : worst) printf("%.6f ", w);
    printf("%.6f ", pw);
    printf("%.6f\n", q);
}
"""


@pytest.fixture(scope="module")
def errors(tmp_path_factory):
    d = tmp_path_factory.mktemp("series")
    src, exe = d / "series.cpp", d / "series"
    src.write_text(HARNESS)
    # series.cuh says what it fuses: no contraction of its own by the compiler
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    return [float(v) for v in subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()]


@pytest.mark.parametrize("k,what,bound", [(0, "reciprocal", 0.501), (1, "root", 0.501), (2, "reciprocal root", 0.501),
                                          (3, "root, short form", 0.751), (4, "reciprocal root, short form", 1.001)])
def test_fp64_series(errors, k, what, bound):
    assert 0.4 < errors[k] <= bound, what


def test_fp32_quotient(errors):
    """Half an ulp for the last rounding; the remainder (exact by fma) times an
    estimate 1.2e-7 off, of a correction of up to 2 ulp, is below 1e-6 ulp: 0.501."""
    assert 0.4 < errors[6] <= 0.501


def test_fp32_scaled_power(errors):
    """Half an ulp for the last addition; what is carried along is of the size of
    the products' roundings (five of 2^-24) and itself rounded: below 1e-5 ulp."""
    assert 0.4 < errors[5] <= 0.501
