// float32 <-> float64 by integer operations.  A conversion instruction occupies the float64 pipe like a
// float64 addition does (2 per clock and SM, 1/64 of the issue slots), while the integer pipes of the
// kernels that convert are idle.  Both functions give the IEEE conversion (round to nearest, ties to even)
// of the values that f32_plain / f64_plain accept: zeros and those that are normal numbers on both sides;
// the callers leave the others to the instruction.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define OPG_HD __host__ __device__ __forceinline__
#else
#define OPG_HD inline
#endif

namespace opg {

struct Bits64 {
    uint32_t hi, lo;
};

// zero or a normal float32
OPG_HD bool f32_plain(uint32_t b) { return (b & 0x7FFFFFFFu) == 0 || ((b >> 23) & 0xFFu) - 1u < 254u; }
OPG_HD Bits64 f32_to_f64_bits(uint32_t b) {
    Bits64 r;
    const uint32_t m = b & 0x7FFFFFFFu;
    r.hi = m == 0 ? b : (b & 0x80000000u) | ((m >> 3) + (896u << 20));
    r.lo = b << 29;
    return r;
}

// zero, or a float64 whose exponent is a normal float32's (rounding up past the largest gives infinity, as
// the conversion does)
OPG_HD bool f64_plain(uint32_t hi, uint32_t lo) {
    return ((hi & 0x7FFFFFFFu) | lo) == 0 || ((hi >> 20) & 0x7FFu) - 897u < 254u;
}
OPG_HD uint32_t f64_to_f32_bits(uint32_t hi, uint32_t lo) {
    const uint32_t m = hi & 0x7FFFFFFFu;
    // exponent and the upper 23 bits of the fraction; half a unit less one bit and the last bit kept round
    const uint32_t t = ((m - (896u << 20)) << 3) | (lo >> 29), rem = lo & 0x1FFFFFFFu;
    const uint32_t up = (rem + 0x0FFFFFFFu + (t & 1u)) >> 29;
    return (hi & 0x80000000u) | ((m | lo) == 0 ? 0u : t + up);
}

}  // namespace opg
