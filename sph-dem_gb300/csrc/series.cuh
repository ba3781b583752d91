/*
 * Quotients, reciprocals and roots from a hardware estimate, by one step of a
 * power series or one remainder, and powers with their rounding errors carried
 * along: plain arithmetic, for the device and, so that the errors can be checked
 * against wider arithmetic, for the host.
 */
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define SPHDEM_HD __host__ __device__ __forceinline__
#else
#define SPHDEM_HD inline
#endif

namespace sphdem {

/* 1/x from an FP32 estimate y (relative error d ~ 1e-7): 1/x = y (1 + e + e^2 +
 * ..), e = 1 - x y, of which d^3 is left; e is rounded once, so the result is
 * good to 0.5 ulp like a division */
SPHDEM_HD double rcp_series(double x, double y) {
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

/* sqrt(x) and, where asked, 1/sqrt(x), from an FP32 estimate y of 1/sqrt(x): one
 * step of the series 1/sqrt(1 - e) = 1 + e/2 + 3 e^2/8 + .., e = 1 - x y^2.  The
 * rounding of x y enters halved: the root to 0.75 ulp, its reciprocal to 1.  For the fluid's sums of tens of
 * pairs, whose error against 64 bits is the same with roots to 0.5 ulp (dam break
 * of 23,018 6.4e-14, of 1,418 3.4e-14) while those cost a step 1 to 3 %. */
SPHDEM_HD double sqrt_series(double x, double y, double *inv = nullptr) {
    const double s = x * y, e = fma(-s, y, 1.0), k = e * fma(e, 0.375, 0.5);
    if (inv) *inv = fma(y, k, y);
    return fma(s, k, s);
}

/* The same to 0.5 ulp: y^2 of an FP32 number is exact, so 1/sqrt(x) rounds once;
 * sqrt(x) = s + (x - s^2) y (1/2 + 3 e/8), whose remainder takes the rounding of
 * s = x y back. */
SPHDEM_HD double sqrt_series_full(double x, double y, double *inv) {
    const double e = fma(-x, y * y, 1.0), k = fma(e, 0.375, 0.5), s = x * y;
    *inv = fma(y, e * k, y);
    return fma(fma(-s, s, x) * y, k, s);
}

/* (g + glo) x^N to 0.5 ulp, the products' rounding errors carried along in FP32
 * (FP64 products in the packing of 1.08 M particles cost 0.019 ms a step) */
template <int N>
SPHDEM_HD float scaled_power(float x, float g, float glo) {
    float p = x, e = 0.f;
    for (int k = 1; k < N; k++) {
        const float q = p * x;
        e = fmaf(e, x, fmaf(p, x, -q));
        p = q;
    }
    const float t = g * p;
    return t + (fmaf(g, p, -t) + fmaf(g, e, glo * p));
}

/* num / den from an estimate y of 1/den (FP32 scalars or pairs), the remainder
 * of the quotient taken back once: 0.5 ulp, where num y by itself is off by up to
 * two.  For numbers whose quotient is in range; infinities give NaN. */
SPHDEM_HD float fused(float a, float b, float c) { return fmaf(a, b, c); }
SPHDEM_HD float times(float a, float b) { return a * b; }
SPHDEM_HD float minus(float a) { return -a; }
#ifdef __CUDACC__
__device__ __forceinline__ float2 fused(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 times(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 minus(float2 a) { return make_float2(-a.x, -a.y); }
#endif
template <class V>
SPHDEM_HD V quotient(V num, V den, V y) {
    const V q = times(num, y);
    return fused(fused(minus(q), den, num), y, q);
}

}  // namespace sphdem
