// k1_math.cuh -- short FP64 reciprocal, reciprocal square root and e^{ix} of the far-field
// sum (k1_fp64.cu), for translation units built with -fmad=false.  A test compares them
// with CUDA's own functions and with 80-bit arithmetic over the ranges that the sum uses.
#pragma once
#include <math.h>

namespace pbt {

// 1/x and 1/sqrt(x) for normal x (rsqrt_n: positive), from the hardware's FP64 seeds y
// (PTX rcp.approx and rsqrt.approx, about 20 bits) and one step of third order: with
// e = 1 - x y, 1/x = y / (1 - e) = y (1 + e + e^2 + ...), the geometric series, and with
// e = 1 - x y^2, 1/sqrt(x) = y (1 - e)^(-1/2) = y (1 + e/2 + 3 e^2/8 + ...), the binomial
// series, each cut after e^2 (Householder's iteration of order two; Newton's is the cut
// after e).  What is left out is below 2^-58 of the result.  Relative errors: half a unit in
// the last place for rcp_n; for rsqrt_n a quarter more, from x y rounded once.
__device__ __forceinline__ double rcp_n(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ double rsqrt_n(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-(x * y), y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}

// e^{ix} from a table of the 128th roots of unity and short polynomials (table look-up as
// in P. T. P. Tang's elementary functions, ACM TOMS 15 and 16): x = n h + r, h = 2 pi /
// 128 in two parts (W. J. Cody and W. Waite's reduction, each product fused, so r is good to
// 1e-16 absolute for |x| < 2^30), and e^{ir} on |r| <= h/2 from minimax fits (E. Y. Remez's
// exchange in 50 digits: 3e-17 for sin, 3e-20 for cos - 1).  15 FP64 operations; the quadrant
// form with polynomials to r^13 and r^14 takes 20 and as many selects and sign changes again,
// the library's checks for huge arguments too and reads its coefficients from memory.
constexpr int kRoots = 128;
__device__ __forceinline__ double reduce_n(double x, int *n32) {
    const double t = fma(x, 20.371832715762604, 6755399441055744.0);
    *n32 = __double2loint(t);  // n modulo 2^32
    const double n = t - 6755399441055744.0;
    return fma(-n, 1.9135106236677394e-18, fma(-n, 0.04908738521234052, x));
}
// e^{i (x + nk h)}, roots[k] = (cos, sin)(k h)
__device__ __forceinline__ void sincos_n(double x, int nk, const double2 *roots, double *sn, double *cs) {
    int n;
    const double r = reduce_n(x, &n);
    const double2 w = roots[(n + nk) & (kRoots - 1)];
    const double z = r * r;
    const double s = fma(r * z, fma(z, 0.008333155366073453, -0.16666666662958388), r);
    const double c = z * fma(z, fma(z, -0.0013888601850806472, 0.041666666656641586), -0.499999999999999);
    *cs = fma(-w.y, s, fma(w.x, c, w.x));
    *sn = fma(w.x, s, fma(w.y, c, w.y));
}

}  // namespace pbt
