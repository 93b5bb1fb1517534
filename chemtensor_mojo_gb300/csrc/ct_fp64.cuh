// FP64 scalars on a kernel's critical path: a division takes 660 cycles on this part and a square
// root ~870, against 65 for an FMA.
#pragma once

namespace ct_fp64 {

// Biased exponent field of x.
__device__ __forceinline__ int exp_field(double x) { return (int)((__double_as_longlong(x) >> 52) & 0x7ff); }
// The mantissa of a normal x as a float in [1, 2), truncated, with x's sign: integer instructions.
__device__ __forceinline__ float mant_f32(double x) {
    const long long b = __double_as_longlong(x);
    return __int_as_float((int)((b >> 63) & 1) << 31 | 127 << 23 | (int)((b >> 29) & 0x7fffff));
}
// A normal float as a double times 2^e, by its bits (the result must be normal).
__device__ __forceinline__ double widen(float x, int e) {
    const int b = __float_as_int(x);
    const long long m = ((long long)(b & 0x7fffffff) << 29) + ((long long)(1023 - 127 + e) << 52);
    return __longlong_as_double(m | ((long long)(b >> 31) << 63));
}
// exponent fields for which the scalings below and the residuals stay normal
__device__ __forceinline__ bool mid_exp(int e) { return (unsigned)(e - 400) < 1248u; }

// Correctly rounded n / d and sqrt(x) from FP32 estimates: one third-order Newton step (to the
// last bit or so), then Markstein's correction with the exact residual (P. W. Markstein,
// Computation of elementary functions on the IBM RISC System/6000 processor, IBM J. Res. Dev.
// 34, 1990), in 6 and 7 dependent operations; outside the middle of the exponent range, and for the
// mantissas below, the plain operators.  (390 and 455 cycles against 660 and ~870.)
//
// Why that rounds correctly.  Estimates are within 2 units in the last place, a relative 1.5 2^-22 with
// the truncated mantissa, so y = 1 / d (1 + c), |c| <= d 2^-54 (1 + h) for d in [1, 2) with h = 2^-10 from
// the cube of that.  The corrected quotient is off by |n / d - q| |c| before its rounding.  Where n / d
// is near the middle of two doubles it is j / (2 D) units from it, D = 2^52 d and j a non-zero
// integer, and q half a unit (n y is within a unit of n / d): right if d^2 (1 + h) < 4, so for d up to
// 2 - 2^-9.  The corrected root is off by (e^2 + 4 e) / (2 m) units, m the root in [2^52, 2^53) and
// e <= 1.1 that of g1; sqrt(x) is (j - 1/4) / (2 m) units from the middle next to m, j an even integer
// with m (m + 1) + j = 0 modulo 2^52 or 2^53.  Those with |j| <= 12 are few, and only x = 2^(2 i) (2 - 2^-52)
// 2 comes out wrong for some estimate.
__device__ __forceinline__ double rcp_near(double d) {   // d's exponent in the middle
    const double y0 = widen(__fdividef(1.0f, mant_f32(d)), 1023 - exp_field(d));
    const double e = fma(-d, y0, 1.0);
    return fma(y0, fma(e, e, e), y0);
}
__device__ __forceinline__ double div_with(double n, double d, double y) {   // y = rcp_near(d)
    const double q = n * y;
    return fma(fma(-d, q, n), y, q);
}
__device__ __forceinline__ bool div_mid(double n, double d) {   // within the middle of the range, d <= 2 - 2^-9
    const int en = exp_field(n), ed = exp_field(d);
    const bool top = ((__double_as_longlong(d) >> 43) & 0x1ff) == 0x1ff;
    return mid_exp(en) && mid_exp(ed) && mid_exp(en - ed + 1023) && !top;
}
__device__ __forceinline__ double div_rn(double n, double d) {
    if (!div_mid(n, d)) return n / d;
    return div_with(n, d, rcp_near(d));
}
__device__ __forceinline__ double sqrt_rn(double x) {
    const int ex = exp_field(x);
    const bool ones = ((__double_as_longlong(x) + 1) & ((1ll << 52) - 1)) == 0;   // an all-ones mantissa
    if (!mid_exp(ex) || x < 0.0 || ones) return sqrt(x);
    // x = m 2^(2k), m in [1, 4)
    const int k = (ex - 1023) >> 1;
    const float mf = mant_f32(x) * (((ex - 1023) & 1) ? 2.0f : 1.0f);
    const double y = widen(rsqrtf(mf), -k);
    const double h = __longlong_as_double(__double_as_longlong(y) - (1ll << 52));   // y / 2
    const double g = x * y;
    const double r = fma(-g, h, 0.5);
    const double p = fma(1.5 * r, r, r);
    const double g1 = fma(g, p, g), h1 = fma(h, p, h);
    return fma(fma(-g1, g1, x), h1, g1);
}

}  // namespace ct_fp64
