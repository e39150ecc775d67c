// el_div.cuh -- FP64 quotients for the WENO6 advection, whose bound is the FP64 pipe.
#pragma once

#include <cuda_runtime.h>

#include <limits>

namespace el {

__device__ __forceinline__ float rcp_approx(float v) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

// num / den (den a positive normal double) in five FP64 operations instead of the nine of a
// division: a float reciprocal of the leading bits, one Newton step, and one correction by the
// residual (P. Markstein, IBM J. Res. Dev. 34, 1990); within an ulp.  Outside the floats' range the
// division itself.
__device__ __forceinline__ bool in_float_range(double v) {  // 2^-120 <= v < 2^120
    return (unsigned)(__double2hiint(v) - 0x38700000) < 0x0f000000u;
}
__device__ __forceinline__ double rcp_newton(double v) {
    const float f = __int_as_float(__funnelshift_l(__double2loint(v), __double2hiint(v) - 0x38000000, 3));
    const unsigned b = (unsigned)__float_as_int(rcp_approx(f));
    const double r = __hiloint2double((int)((b >> 3) + 0x38000000u), (int)(b << 29));
    return fma(r, fma(-v, r, 1.0), r);  // 44 bits
}
__device__ __forceinline__ double div_newton(double num, double den) {
    if (!in_float_range(den)) return num / den;
    const double r = rcp_newton(den), q = num * r;
    return fma(fma(-den, q, num), r, q);
}
// 1 / v to within an ulp (one more Newton step); NaN for a product that overflowed, whose 0 would silently
// drop the weights formed with it (the result's NaN then takes the general path)
__device__ __forceinline__ double inverse(double v) {
    if (!in_float_range(v)) return v <= std::numeric_limits<double>::max() ? 1.0 / v : std::numeric_limits<double>::quiet_NaN();
    const double r = rcp_newton(v);
    return fma(r, fma(-v, r, 1.0), r);
}

}  // namespace el
