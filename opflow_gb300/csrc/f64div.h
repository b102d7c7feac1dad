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

// a / b, correctly rounded, given y = 1/b to within an ulp (recip_fast): q = a y, the remainder r = a - q b, and
// q + r y (the division steps of Markstein, IBM J. Res. Dev. 34 (1990)).  q is off a / b by less than 1.6 ulps of q
// and y by 2^-52 of 1/b, so q + r y is off a / b by less than 2^-51 ulp before its rounding; it is rounded to a / b's neighbour
// unless a / b lies that near the middle of two numbers.  That is looked for on the bits (integer operations,
// which cost next to nothing here): |r| near ulp(q) b / 2 or 3 ulp(q) b / 2, or q next to a power of two (below
// it the numbers are denser); then, and where an exponent is near the ends of the range, the lanes concerned
// divide.  SIGNED: operands of either sign and zero numerators (else positive ones, or the division apart).
template <bool SIGNED>
__device__ __forceinline__ double div_rn(double a, double b, double y) {
    constexpr unsigned long long MAG = 0x7FFFFFFFFFFFFFFFull, FRAC = 0xFFFFFFFFFFFFFull, ONE = 0x10000000000000ull;
    const double q = __dmul_rn(a, y);
    const double r = __fma_rn(-q, b, a);
    double v = __fma_rn(r, y, q);
    unsigned long long ab = (unsigned long long) __double_as_longlong(a), bb = (unsigned long long) __double_as_longlong(b),
                       qb = (unsigned long long) __double_as_longlong(q);
    const unsigned long long rb = (unsigned long long) __double_as_longlong(r) & MAG;
    if (SIGNED) {
        ab &= MAG;
        bb &= MAG;
        qb &= MAG;
    }
    const unsigned ea = (unsigned) (ab >> 52), eb = (unsigned) (bb >> 52), eq = (unsigned) (qb >> 52);
    bool bad = ea - 200u > 1600u || eq - 200u > 1600u;
    bad |= (qb & FRAC) < 3;
    // T = ulp(q) b / 2
    const unsigned long long T = bb + ((unsigned long long) eq << 52) - ((unsigned long long) (1023 + 53) << 52);
    bad |= rb - T + 64 <= 128;
    // |r| against 3 T: significands 2^k m(r) and 3 m(b), k the difference of the exponents
    const int k = (int) (rb >> 52) - (int) (T >> 52);
    const unsigned long long mr = ((rb & FRAC) | ONE) << (k & 3), mb = 3 * ((bb & FRAC) | ONE);
    bad |= (k == 1 || k == 2) && mr - mb + 256 <= 512;
    if (SIGNED && ab == 0) {
        bad = false;
        v = q;  // (a zero of the right sign)
    }
    bad |= eb - 200u > 1600u;
    if (bad) v = div_apart(a, b);
    return v;
}

// a / b for the smoothers, by the same six operations without the search for the middles: the IEEE quotient but
// for one in 2^50, then its neighbour.  An operand or a quotient near either end of the range is divided.  (With
// div_rn a 192^3 float64 solve takes 33.9 instead of 31.0 ms: its integer operations are not free there.)
__device__ __forceinline__ double quotient(double a, double b) {
    const double y = recip_fast(b), q = __dmul_rn(a, y);
    double v = __fma_rn(__fma_rn(-q, b, a), y, q);
    auto ends = [](double x) { return (unsigned) (((__double2hiint(x) >> 20) & 0x7FF) - 200) > 1600u; };
    const bool zero = ((__double2hiint(a) & 0x7FFFFFFF) | __double2loint(a)) == 0;
    v = zero ? q : v;  // (a zero of the right sign)
    if (ends(b) || (!zero && (ends(a) || ends(q)))) v = div_apart(a, b);
    return v;
}
__device__ __forceinline__ float quotient(float a, float b) { return a / b; }

}  // namespace opg
