// The exact FTCS update u + s * (d2<0>(u) + d2<1>(u) [+ d2<2>(u)]) on a uniform mesh: warps march strips
// of a 2D or 3D box with the reference's IEEE operations in its order (D2SecondOrderCentered::eval,
// D2SecondOrderCentered.hpp:160-171, summed in tree order, then u + s * sum), bit-identical to it.
//
// What bounds it is the float64 pipe (2 operations per clock and SM, 1/64 of the issue slots), so the
// float64 operations are what is saved:
//  - the one-sided difference (u(i+1) - u(i)) / h of a face is the right one of cell i and the left one of
//    cell i + 1: it is formed once, the left lane's taken by a shuffle (x), the last row's (y) or the last
//    plane's (z) kept in a register;
//  - x / h for a power of two h moves the exponent field (no float64 instruction); zeros stay, and a warp
//    that holds a subnormal or non-finite operand or result takes the float64 multiply;
//  - x / h for any other h is fma(x, ch, x * cl) with ch + cl = 1/h to 106 bits, two operations.  The host
//    finds the significands of x for which that is not the IEEE quotient (none, seldom one: div2_failures
//    in stencil.cu); a warp that holds one divides.
// Operations per cell, 2D / 3D: 7 / 10 for a power of two, 15 / 22 otherwise, against 9 / 13 and 27 / 40
// with every difference formed per cell and three operations per division (and the skipped side of each
// division's branches); two of a warp's 32 columns
// only supply neighbours.  Measured per step: 1025^2 47.5 -> 20.4 us (the pipe takes an addition every
// 19 cycles at best: 16.2 us), 301 x 257 x 333 (one power of two) 2074 -> 1010 us, 64 grids of 4.35 M points
// 226 -> 158 us.
#pragma once
#include "f64div.h"
#include "stencil.h"

namespace opg {

constexpr int EX_COLS = 30;    // columns a warp updates (lanes 1..30; lanes 0 and 31 supply neighbours)
constexpr int EX_ROWS = 4;     // 3D: rows a warp updates
constexpr int EX_WARPS = 4;
// Tiles per SM a launch has at least, where the box allows (12 to 192 tried): 2D the same from 12 on, 3D
// 301 x 257 x 333 4.26 ms per 4 steps with 12 and 24, 4.05 with 48 (shorter marches even out the last wave).
constexpr int EX_FILL = 24, EX_FILL3 = 48;

// The dims whose h is a power of two, bit d for dim d: a template parameter of the kernels.
inline int exact_mode(const AxisParams& P) {
    int m = 0;
    for (int d = 0; d < P.ndim; ++d) m |= P.pow2[d] ? 1 << d : 0;
    return m;
}

// The rare cases in functions of their own: of such a branch within the code the compiler issues both
// sides under predicates, and a float64 operation that is predicated off takes its 16 cycles of the pipe
// all the same (measured).
static __device__ __noinline__ double mul_apart(double x, double y) { return __dmul_rn(x, y); }

// correctly rounded x / h[D], called by whole warps
template <int PM, int D>
__device__ __forceinline__ double div_exact(double x, const AxisParams& P) {
    const int hi = __double2hiint(x), lo = __double2loint(x);
    if constexpr ((PM & (1 << D)) != 0) {
        const int e = (hi >> 20) & 0x7FF, k = P.shift[D];
        const bool zero = ((hi & 0x7FFFFFFF) | lo) == 0;
        const bool special = !zero && ((unsigned) (e - 1) >= 2046u || (unsigned) (e + k - 1) >= 2046u);
        double r = __hiloint2double(zero ? hi : hi + k * (1 << 20), lo);
        if (__any_sync(0xffffffffu, special)) {
            const double m = mul_apart(x, P.inv_h[D]);
            r = special ? m : r;
        }
        return r;
    } else {
        double r = __fma_rn(x, P.inv_h[D], __dmul_rn(x, P.cl[D]));
        if (P.guard[D]) {
            const bool bad = lo == P.bad_lo[D] && (hi & 0xFFFFF) == P.bad_hi[D];
            if (__any_sync(0xffffffffu, bad)) {
                const double m = div_apart(x, P.h[D]);
                r = bad ? m : r;
            }
        }
        return r;
    }
}

// Rows [ys, ye) of the columns x0 .. x0 + EX_COLS - 1 of a 2D box; PM: exact_mode.  Loads run two rows
// ahead.
template <int PM>
__device__ __forceinline__ void exact_strip2(const FieldView& in, const FieldView& out, const Box& box, const AxisParams& P, int x0, int ys, int ye) {
    const int lane = threadIdx.x & 31;
    const int i = x0 - 1 + lane, ic = min(i, box.hi[0]), jmax = box.hi[1];
    const bool vx = lane >= 1 && lane <= EX_COLS && i < box.hi[0];
    const double* src = in.data + (ic - in.off[0]) - (long long) in.off[1] * in.sy + (long long) (box.lo[2] - in.off[2]) * in.sz;
    double* dst = out.data + (i - out.off[0]) + (long long) (ys - out.off[1]) * out.sy + (long long) (box.lo[2] - out.off[2]) * out.sz;
    const double* p = src + (long long) (ys - 1) * in.sy;
    const double below = p[0];
    double c = p[in.sy], n1 = p[2 * in.sy], n2 = src[(long long) min(ys + 2, jmax) * in.sy];
    double fy = div_exact<PM, 1>(__dsub_rn(c, below), P);
    for (int j = ys; j < ye; ++j) {
        const double up = n1;
        n1 = n2;
        n2 = src[(long long) min(j + 3, jmax) * in.sy];
        const double fyu = div_exact<PM, 1>(__dsub_rn(up, c), P);
        const double d2y = div_exact<PM, 1>(__dsub_rn(fyu, fy), P);
        const double fx = div_exact<PM, 0>(__dsub_rn(__shfl_down_sync(0xffffffffu, c, 1), c), P);
        const double d2x = div_exact<PM, 0>(__dsub_rn(fx, __shfl_up_sync(0xffffffffu, fx, 1)), P);
        const double v = __dadd_rn(c, __dmul_rn(P.s, __dadd_rn(d2x, d2y)));  // (a sum of two does not depend on their order)
        if (vx) *dst = v;
        dst += out.sy;
        fy = fyu;
        c = up;
    }
}

// Planes [zs, ze) of EX_COLS columns from x0 and EX_ROWS rows from y0 of a 3D box; the next plane is on
// its way while a plane is updated.
template <int PM>
__device__ __forceinline__ void exact_strip3(const FieldView& in, const FieldView& out, const Box& box, const AxisParams& P, int x0, int y0, int zs,
                                             int ze) {
    constexpr int R = EX_ROWS;
    const int lane = threadIdx.x & 31;
    const int i = x0 - 1 + lane, ic = min(i, box.hi[0]);
    const bool vx = lane >= 1 && lane <= EX_COLS && i < box.hi[0];
    const double* src = in.data + (ic - in.off[0]) - (long long) in.off[2] * in.sz;
    double* dst = out.data + (i - out.off[0]) + (long long) (y0 - out.off[1]) * out.sy + (long long) (zs - out.off[2]) * out.sz;
    long long row[R + 2];  // rows y0 - 1 .. y0 + R, clamped to the farthest row the stencil reads
#pragma unroll
    for (int r = 0; r < R + 2; ++r) row[r] = (long long) (min(y0 - 1 + r, box.hi[1]) - in.off[1]) * in.sy;
    double cur[R + 2], nxt[R + 2], fz[R];
    {
        const double* p = src + (long long) zs * in.sz;
#pragma unroll
        for (int r = 0; r < R + 2; ++r) {
            cur[r] = p[row[r]];
            nxt[r] = p[row[r] + in.sz];
        }
#pragma unroll
        for (int r = 0; r < R; ++r) fz[r] = div_exact<PM, 2>(__dsub_rn(cur[r + 1], p[row[r + 1] - in.sz]), P);
    }
    const int last = P.order[2];  // the term added last (the first two commute)
    for (int k = zs; k < ze; ++k) {
        double ahead[R + 2];
        const double* p = src + (long long) min(k + 2, box.hi[2]) * in.sz;
#pragma unroll
        for (int r = 0; r < R + 2; ++r) ahead[r] = p[row[r]];
        double fy = div_exact<PM, 1>(__dsub_rn(cur[1], cur[0]), P);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const double c = cur[r + 1];
            const double fyu = div_exact<PM, 1>(__dsub_rn(cur[r + 2], c), P);
            const double d2y = div_exact<PM, 1>(__dsub_rn(fyu, fy), P);
            fy = fyu;
            const double fx = div_exact<PM, 0>(__dsub_rn(__shfl_down_sync(0xffffffffu, c, 1), c), P);
            const double d2x = div_exact<PM, 0>(__dsub_rn(fx, __shfl_up_sync(0xffffffffu, fx, 1)), P);
            const double fzu = div_exact<PM, 2>(__dsub_rn(nxt[r + 1], c), P);
            const double d2z = div_exact<PM, 2>(__dsub_rn(fzu, fz[r]), P);
            fz[r] = fzu;
            const double a = last == 0 ? d2y : d2x, b = last == 2 ? d2y : d2z, e = last == 0 ? d2x : (last == 1 ? d2y : d2z);
            const double v = __dadd_rn(c, __dmul_rn(P.s, __dadd_rn(__dadd_rn(a, b), e)));
            if (vx && y0 + r < box.hi[1]) dst[r * out.sy] = v;
        }
        dst += out.sz;
#pragma unroll
        for (int r = 0; r < R + 2; ++r) {
            cur[r] = nxt[r];
            nxt[r] = ahead[r];
        }
    }
}

// A warp's tile of an exact update: 2D: rows [a, b) of the columns from x0; 3D: planes [a, b) of the
// columns from x0 and the rows from y0.
struct ExactTile {
    int item;
    int x0, y0, a, b;
};
template <int PM, int ND>
__device__ __forceinline__ void exact_tile(const FieldView& in, const FieldView& out, const Box& box, const AxisParams& P, const ExactTile& T) {
    if constexpr (ND == 2) exact_strip2<(PM & 3)>(in, out, box, P, T.x0, T.a, T.b);
    else exact_strip3<PM>(in, out, box, P, T.x0, T.y0, T.a, T.b);
}
// calls f(std::integral_constant<int, mode>) for the mode of exact_mode
template <typename F>
__host__ __device__ __forceinline__ void exact_dispatch(int mode, F&& f) {
    switch (mode) {
#define OPG_EXACT_CASE(M) case M: f(std::integral_constant<int, M>{}); break;
        OPG_EXACT_CASE(0) OPG_EXACT_CASE(1) OPG_EXACT_CASE(2) OPG_EXACT_CASE(3) OPG_EXACT_CASE(4) OPG_EXACT_CASE(5) OPG_EXACT_CASE(6)
#undef OPG_EXACT_CASE
        default: f(std::integral_constant<int, 7>{}); break;
    }
}

// Marching length (rows in 2D, planes in 3D) of the tiles of a box: the longest of at most 32 that leaves
// the box `share` of a launch's tiles, at least 4.
inline int exact_march(const Box& box, int ndim, int sms, double share) {
    const long long want = (long long) (share * sms * (ndim == 3 ? EX_FILL3 : EX_FILL));
    const long long nx = box.hi[0] - box.lo[0], ny = box.hi[1] - box.lo[1], nz = box.hi[2] - box.lo[2];
    const long long across = std::max(1LL, (nx + EX_COLS - 1) / EX_COLS * (ndim == 3 ? (ny + EX_ROWS - 1) / EX_ROWS : 1));  // (an empty box has none)
    const long long len = ndim == 3 ? nz : ny;
    const long long runs = std::max(1LL, (want + across - 1) / across);
    return (int) std::max(4LL, std::min(32LL, (len + runs - 1) / runs));
}

}  // namespace opg
