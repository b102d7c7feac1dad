// Float64 reciprocals and quotients from fused operations: the float64 pipe takes 16 cycles per warp
// operation, and the compiler's division is a dozen of them.
#pragma once

namespace opg {

// 1/x for x in the normal range: the hardware's approximate reciprocal refined by the cubic Newton step
// y = r + r*(e + e^2), e = 1 - x*r (Newton-Raphson iteration for 1/x with the second-order term; the
// relative error goes from eps to about eps^3).
__device__ __forceinline__ double recip_fast(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double e = __fma_rn(-x, r, 1.0);
    return __fma_rn(__fma_rn(e, e, e), r, r);
}

// The division for the operands that the steps built on recip_fast leave out, apart: a float64 operation
// that is predicated off takes the pipe's time all the same.
static __device__ __noinline__ double div_apart(double a, double b) { return __ddiv_rn(a, b); }

// a / b in six operations: q = a y with y = 1/b, the remainder r = a - q b, q + r y (Markstein, IBM J. Res.
// Dev. 34 (1990)): off the quotient by less than 2^-50 ulp before its rounding.  A b, or a quotient, near
// either end of the range is divided.
__device__ __forceinline__ double quotient(double a, double b) {
    const double y = recip_fast(b), q = __dmul_rn(a, y);
    double v = __fma_rn(__fma_rn(-q, b, a), y, q);
    const int eb = (__double2hiint(b) >> 20) & 0x7FF, ea = (__double2hiint(a) >> 20) & 0x7FF;
    if ((unsigned) (eb - 200) > 1600u || ((unsigned) (ea - 200) > 1600u && ((__double2hiint(a) & 0x7FFFFFFF) | __double2loint(a)) != 0)) v = div_apart(a, b);
    return v;
}
__device__ __forceinline__ float quotient(float a, float b) { return a / b; }

}  // namespace opg
