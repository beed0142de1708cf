// devmath.cuh -- small device math helpers shared by the kernels.
#pragma once
#include <cuda_runtime.h>

namespace psb {

// 1/d without special-case branches, for finite normal d: the PTX
// rcp.approx.ftz.f64 estimate refined by two Newton-Raphson steps for the
// reciprocal, r <- r + r (1 - d r), each of which doubles the number of
// correct bits.  Agrees with the correctly rounded 1.0 / d to within one unit
// in the last place (checked by the test suite) where it is used: mu + mu0 of
// visible facets, in (2e-8, 2], and counts of points.  Zero and negative sums
// also come in, of facets out of sight in the brightness sweep, where the
// result (a NaN for zero) is dropped.
__device__ __forceinline__ double rcp_approx(double d)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    return r;
}

__device__ __forceinline__ double rcp_step(double d, double r)
{
    return fma(r, fma(-d, r, 1.0), r);
}

__device__ __forceinline__ double rcp_nr(double d)
{
    return rcp_step(d, rcp_step(d, rcp_approx(d)));
}

}  // namespace psb
