/*
 * fp64.cuh -- FP64 square root and division by a known constant without
 * branches, for the dependent chains of the sweep kernels (a branch per root
 * keeps the compiler from interleaving a thread's independent chains).
 *
 * Both end in the residual correction of Markstein ("Software division and
 * square root using Goldschmidt's algorithms", 2004): the residual of a
 * result within one ulp is exact in one multiply-add, and its correction
 * rounds to the IEEE result (in 1.2e9 random arguments each, 139 roots were
 * one ulp off and no quotient).  The root takes 68 cycles of a dependent
 * chain, sqrt() 82.
 */
#pragma once
#include <cuda_runtime.h>

namespace fk64 {

/* Whether sqrt64(x) is the square root of x (NaN for x < 0): false for
 * zero, tiny, huge, infinite and NaN arguments. */
__device__ __forceinline__ bool sqrt64_ok(double x) { return x < 0.0 || (x > 1e-280 && x < 1e280); }

/* sqrt(x) where sqrt64_ok(x).  With y ~ 1 / sqrt(x) (the hardware's
 * approximation) and e = 1 - x y^2, Householder's third-order step gives
 * x y (1 + e (1/2 + 3/8 e)), then the residual correction. */
__device__ __forceinline__ double sqrt64(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double t = x * y;
    const double e = fma(-t, y, 1.0);
    const double g = fma(e * t, fma(0.375, e, 0.5), t);
    return fma(fma(-g, g, x), 0.5 * y, g);
}

/* a / c with ci = 1 / c (rounded): the IEEE quotient for normal quotients. */
__device__ __forceinline__ double div64(double a, double c, double ci)
{
    const double q = a * ci;
    return fma(fma(-q, c, a), ci, q);
}

} // namespace fk64
