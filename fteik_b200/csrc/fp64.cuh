/*
 * fp64.cuh -- FP64 square root and division by a known constant without
 * branches, for the dependent chains of the sweep kernels (a branch per root
 * keeps the compiler from interleaving a thread's independent chains).
 *
 * Both end in the residual correction of Markstein ("Software division and
 * square root using Goldschmidt's algorithms", 2004): the residual of a
 * result within one ulp is exact in one multiply-add, and its correction
 * rounds to the IEEE result if the factor of the correction is good to the
 * last bits (a factor good to 22 bits leaves one root in 10^7 an ulp off, one
 * good to 44 still some of those next to the middle of two numbers).  Equal to
 * sqrt() and the division for all arguments whose result lies closer to the
 * middle of two numbers than the factor's error reaches, and for random ones.
 * The root takes 71 cycles of a dependent chain, sqrt() 78; its factor is formed
 * beside the chain without a further FP64 operation (the half of y in integers,
 * the step w shared with the root): with one more, 256 2D sources on 151 x 301
 * take 3.30 ms instead of 2.95.
 */
#pragma once
#include <cuda_runtime.h>

namespace fk64 {

/* Whether sqrt64(x) is the square root of x (NaN for x < 0): false for
 * zero, tiny, huge, infinite and NaN arguments. */
__device__ __forceinline__ bool sqrt64_ok(double x) { return x < 0.0 || (x > 1e-280 && x < 1e280); }

/* sqrt(x) where sqrt64_ok(x).  With y ~ 1 / sqrt(x) (the hardware's
 * approximation) and e = 1 - x y^2, Householder's third-order step gives
 * x y (1 + e (1/2 + 3/8 e)) and, for the factor 1 / (2 sqrt(x)) of the residual
 * correction, y / 2 (1 + e (1/2 + 3/8 e)). */
__device__ __forceinline__ double sqrt64(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double hy = __hiloint2double(__double2hiint(y) - (1 << 20), __double2loint(y));   /* y / 2 */
    const double t = x * y;
    const double e = fma(-t, y, 1.0);
    const double w = e * fma(0.375, e, 0.5);
    const double g = fma(w, t, t), h = fma(w, hy, hy);
    return fma(fma(-g, g, x), h, g);
}

/* a / c with ci = 1 / c (rounded): the IEEE quotient for normal quotients. */
__device__ __forceinline__ double div64(double a, double c, double ci)
{
    const double q = a * ci;
    return fma(fma(-q, c, a), ci, q);
}

} // namespace fk64
