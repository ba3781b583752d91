/*
 * Quotients, reciprocals and roots from a hardware estimate, by one step of a
 * power series or one remainder: plain arithmetic, for the device and, so that
 * their errors can be checked against wider arithmetic, for the host.
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

}  // namespace sphdem
