// Fused 2D multigrid steps of the large red-black float32 levels with a class-table operator, marching
// down the rows in registers.
//
// The chunked kernels make one pass over a level per half sweep, residual, restriction and
// prolongation.  Here one warp takes a strip of a level and runs the whole down-leg step on it -
// pre-smoothing from a zero guess, residual, restriction into the next level - or the whole up-leg step
// - prolongation and post-smoothing - in one march along y:
//  - lane l holds the columns 2l and 2l + 1 of 64 consecutive ones, so every half sweep updates exactly
//    one cell per lane and row, the same column parity in every lane, with one warp shuffle for the
//    x-neighbour in the adjacent lane and the y-neighbours in the lane's own registers;
//  - half sweep h works one row behind half sweep h - 1, the residual one row behind the last half
//    sweep, so a step of the march takes one new row through the whole pipeline; the rows in flight sit
//    in a register window that moves on by two rows at a time (a march unrolled by the window's length
//    needs no moves, but its code no longer fits the instruction caches: measured 45 us per launch on
//    levels of any size, against 10 to 24 us);
//  - each half sweep invalidates one more column and row at the strip's edge: the halo is 2 x sweeps
//    cells (one more for node-centred restriction, whose weights reach a neighbouring residual).
// There is no shared memory and no barrier.  Level data crosses memory once per step: down reads b and
// writes the smoothed x and the coarse b, up reads x, b and the coarse x and writes x.
//
// The per-cell arithmetic is the chunked kernels' in their operation order, spelled with the fused
// multiply-adds the compiler forms there, so the two paths give bit-identical iterates.  A neighbour that
// does not exist has coefficient 0 here (the chunked kernels skip its term), a column or row outside the
// level an inverse diagonal of 0, so its x stays 0.
//
// Strips of one launch read their halos from the level's arrays while others write their results, so a
// launch never writes the array it reads: the down step leaves the smoothed x in the level's r array
// (the residual itself stays in registers), the up step reads that array and writes x.
//
// What bounds it: on large levels instruction issue (about 95 warp instructions per row of 64 columns,
// half of the issue slots used; 2.5 warp instructions per cell at 16 rows a strip), on small ones the
// chain of half sweeps within a row (about 500 cycles).  Against the shared-memory tiles of 54 x 32 cells
// it replaced: 2048^2 level 0 down 71 -> 24 us, up 114 -> 27 us; 18.5 M cells of 64 Helmholtz problems down
// 460 -> 95 us, up 757 -> 131 us.
#include "mg_device.h"

namespace opg {

constexpr int STRIP_WARPS = 4;
constexpr int PF = 2;  // rows of loads in flight ahead of the march (even; 4 measured no faster)
constexpr unsigned FULL = 0xffffffffu;

// One column's coefficients in one row class: centre, x-, x+, y-, y+, (z-, z+,) 1 / centre.
struct ColCoef {
    float c0, c1, c2, c3, c4, inv;
};
static_assert(TSTRIDE == 8 && NSLOT == 7, "a class-table row is two 16-byte loads");
__device__ __forceinline__ ColCoef col_coef(const float* __restrict__ row) {
    const float4 a = *(const float4*) row, b = *(const float4*) (row + 4);
    return ColCoef{a.x, a.y, a.z, a.w, b.x, b.w};
}

__device__ __forceinline__ int wrap_pos(int g, int n) {
    g %= n;
    return g < 0 ? g + n : g;
}

// Plain (coherent) loads
__device__ __forceinline__ float ldf(const float* p) { return __ldca(p); }

// off-diagonal sum of the cell in column P (0: even, 1: odd) of a row: W and E from the row's other
// column (P = 0: W in the lane below, P = 1: E in the lane above), S and N from the rows before and after
template <int P>
__device__ __forceinline__ float offdiag(const ColCoef& K, const float (&row)[2], float south, float north) {
    const float w = P == 0 ? __shfl_up_sync(FULL, row[1], 1) : row[0];
    const float e = P == 0 ? row[1] : __shfl_down_sync(FULL, row[0], 1);
    float acc = __fmaf_rn(K.c1, w, 0.f);
    acc = __fmaf_rn(K.c2, e, acc);
    acc = __fmaf_rn(K.c3, south, acc);
    return __fmaf_rn(K.c4, north, acc);
}

// Geometry of a strip.  The chunk holds the strip's own cells: columns i0 .. i0 + cnt, rows j ..
// j + nrows; lane 0's even column is i0 - hx.
struct Strip {
    int n0, n1, per1;
    int ist;          // lane 0's even column
    int jb, je;       // first and last row the march needs (it runs in pairs of rows from jb)
    int j0, j1;       // the strip's own rows [j0, j1)
    int i0, i1;       // its own columns [i0, i1)
    int ge;           // the lane's even column, unwrapped
    int we, wo;       // the lane's columns in the level (wrapped where x is periodic)
    bool oke, oko;    // whether they exist
    const float *te, *to;  // their class-table rows for the first row of the level; columns outside the
                           // level point at all-zero rows (a 2D level's table uses 9 of the 27 classes)
    __device__ __forceinline__ bool row_ok(int r) const { return per1 || (unsigned) r < (unsigned) n1; }
    // row r's row in the level (a strip reaches less than a period beyond a periodic level)
    __device__ __forceinline__ int row_of(int r) const { return per1 ? (r < 0 ? r + n1 : (r >= n1 ? r - n1 : r)) : r; }
};

__device__ __forceinline__ Strip strip_of(const LvlDev& L, const Chunk& C, int hx, int hy, int lane) {
    Strip S;
    S.n0 = L.n[0];
    S.n1 = L.n[1];
    S.per1 = L.per[1];
    S.ist = C.i0 - hx;
    S.j0 = C.j;
    S.j1 = min(C.j + C.nrows, S.n1);
    S.i0 = max(C.i0, 0);
    S.i1 = min(C.i0 + C.cnt, S.n0);
    // row jb's even columns have colour 0, so that a row's colours follow from its distance to jb
    S.jb = C.j - hy;
    S.jb -= (S.ist + S.jb) & 1;
    S.je = min(C.j + C.nrows, (S.n1 + 1) & ~1) - 1 + hy;
    S.ge = S.ist + 2 * lane;
    S.we = L.per[0] ? wrap_pos(S.ge, S.n0) : S.ge;
    S.wo = L.per[0] ? wrap_pos(S.ge + 1, S.n0) : S.ge + 1;
    S.oke = (unsigned) S.we < (unsigned) S.n0;
    S.oko = (unsigned) S.wo < (unsigned) S.n0;
    S.te = L.T32 + (S.oke ? pos_class(S.we, S.n0) : 9) * TSTRIDE;
    S.to = L.T32 + (S.oko ? pos_class(S.wo, S.n0) : 9) * TSTRIDE;
    return S;
}

// How a strip treats the rows at the level's first and last row and beyond.
enum RowMode {
    ROWS_INNER = 0,    // the march never comes near them
    ROWS_DIAG = 1,     // only the centre coefficient differs there (LvlDev::uoff), and beyond them x stays 0 by
                       // an inverse diagonal of 0: selects, no branches
    ROWS_GENERAL = 2,  // every coefficient may differ: read from the class table, rows beyond skipped
};

// one column: the interior rows' coefficients, and centre and inverse in the first and the last row
struct Column {
    ColCoef in;
    float c0f, c0l, invf, invl;
    const float* t;
};
template <int MODE>
__device__ __forceinline__ Column column_of(const float* t) {
    Column K;
    K.t = t;
    K.in = col_coef(t + 3 * TSTRIDE);
    K.c0f = K.c0l = K.invf = K.invl = 0.f;
    if (MODE == ROWS_DIAG) {
        const ColCoef f = col_coef(t), l = col_coef(t + 2 * 3 * TSTRIDE);
        K.c0f = f.c0;
        K.invf = f.inv;
        K.c0l = l.c0;
        K.invl = l.inv;
    }
    return K;
}

// a column's coefficients in row r
template <int MODE>
__device__ __forceinline__ ColCoef row_coef(const Strip& S, int r, const Column& C) {
    ColCoef K = C.in;
    if (MODE != ROWS_INNER) {
        const int w = S.row_of(r);
        if (MODE == ROWS_DIAG) {
            K.inv = w == 0 ? C.invf : (w == S.n1 - 1 ? C.invl : ((unsigned) w < (unsigned) S.n1 ? K.inv : 0.f));
            K.c0 = w == 0 ? C.c0f : (w == S.n1 - 1 ? C.c0l : K.c0);
        } else if (w == 0 || w == S.n1 - 1) {
            K = col_coef(C.t + (w == 0 ? 0 : 2 * 3 * TSTRIDE));
        }
    }
    return K;
}

// The Gauss-Seidel update of row r's column P; X[k] is row r's pair, X[k - 1] and X[k + 1] its neighbours'.
template <int P, int MODE, int NX>
__device__ __forceinline__ void strip_gs(const Strip& S, int r, float (&X)[NX][2], int k, float bv, const Column& Ce, const Column& Co) {
    if (MODE != ROWS_GENERAL || S.row_ok(r)) {
        const ColCoef K = row_coef<MODE>(S, r, P ? Co : Ce);
        X[k][P] = __fmul_rn(__fsub_rn(bv, offdiag<P>(K, X[k], X[k - 1][P], X[k + 1][P])), K.inv);
    }
}

template <int P>
struct Par {
    static constexpr int value = P;
};

// Down-leg step: SW red-black sweeps of A x = b from x = 0, the residual, its restriction into the next
// level (whose x becomes 0).  Rows come in pairs (jp, jp + 1); the windows hold rows jp - LAG - 1 .. jp + 1 of
// x and jp - LAG .. jp + 1 + PF of b (the last PF on their way).
template <int SW, bool NODE, int MODE>
__device__ __forceinline__ void strip_down(const LvlDev& L, const LvlDev& Lc, const Strip& S, int lane) {
    constexpr int LAG = 2 * SW;  // the residual's row lags the newest row by this
    constexpr int NX = LAG + 3, NB = LAG + 2 + PF;
    const Column Ke = column_of<MODE>(S.te), Ko = column_of<MODE>(S.to);
    constexpr bool YIN = MODE == ROWS_INNER;
    const float* bg = L.b32;
    float* xg = L.r32;
    float* bc = Lc.b32;
    float* xc = Lc.x32;
    const int cn0 = Lc.n[0];
    const bool adjoint = L.adjoint;
    const bool own_e = S.ge >= S.i0 && S.ge < S.i1, own_o = S.ge + 1 >= S.i0 && S.ge + 1 < S.i1;
    // (children beyond the level's faces are left out of the restriction, also where it is periodic)
    const bool ein = (unsigned) S.ge < (unsigned) S.n0, oin = (unsigned) (S.ge + 1) < (unsigned) S.n0;
    float X[NX][2], B[NB][2];
#pragma unroll
    for (int k = 0; k < NX; ++k) X[k][0] = X[k][1] = 0.f;
#pragma unroll
    for (int k = 0; k < NB; ++k) B[k][0] = B[k][1] = 0.f;
    auto load = [&](int r, float (&v)[2]) {
        const bool ok = YIN || S.row_ok(r);
        const float* p = bg + (long long) (YIN ? r : (ok ? S.row_of(r) : 0)) * S.n0;
        v[0] = ok && S.oke ? ldf(p + S.we) : 0.f;
        v[1] = ok && S.oko ? ldf(p + S.wo) : 0.f;
    };
    float pa = 0.f;                                    // cell-centred: the even row's part of the coarse sum
    float q1e = 0.f, q1o = 0.f, q2e = 0.f, q2o = 0.f;  // node-centred: the residuals one and two rows back
    auto row = [&](auto par, int j) {
        constexpr int P = decltype(par)::value;  // row j = jp + P; every half sweep of this row's step updates column P
        constexpr int kx = LAG + 1 + P, kb = LAG + P;  // row j in X and B
        // half sweep 1 (colour 0) of row j from the zero guess: x = b / c0
        X[kx][0] = X[kx][1] = 0.f;
        if (MODE != ROWS_GENERAL || S.row_ok(j)) X[kx][P] = __fmul_rn(B[kb][P], row_coef<MODE>(S, j, P ? Ko : Ke).inv);
        // half sweep h of row j - (h - 1)
#pragma unroll
        for (int d = 1; d < LAG; ++d) strip_gs<P, MODE>(S, j - d, X, kx - d, B[kb - d][P], Ke, Ko);
        // the residual of row r, whose x is final
        const int r = j - LAG;
        float re = 0.f, ro = 0.f;
        if (MODE != ROWS_GENERAL || S.row_ok(r)) {
            const ColCoef E = row_coef<MODE>(S, r, Ke), O = row_coef<MODE>(S, r, Ko);
            re = __fsub_rn(B[kb - LAG][0], __fmaf_rn(E.c0, X[kx - LAG][0], offdiag<0>(E, X[kx - LAG], X[kx - LAG - 1][0], X[kx - LAG + 1][0])));
            ro = __fsub_rn(B[kb - LAG][1], __fmaf_rn(O.c0, X[kx - LAG][1], offdiag<1>(O, X[kx - LAG], X[kx - LAG - 1][1], X[kx - LAG + 1][1])));
        }
        if (!ein || !(YIN || (unsigned) r < (unsigned) S.n1)) re = 0.f;
        if (!oin || !(YIN || (unsigned) r < (unsigned) S.n1)) ro = 0.f;
        if (r >= S.j0 && r < S.j1) {
            float* p = xg + (long long) r * S.n0 + S.ge;
            if (own_e) p[0] = X[kx - LAG][0];
            if (own_o) p[1] = X[kx - LAG][1];
        }
        if (!NODE) {
            // (row jb and lane 0's even column are even, so rows 2 I and 2 I + 1 come as one pair)
            if (P == 0) {
                pa = __fadd_rn(re, ro);
            } else if (own_e && r - 1 >= S.j0 && r - 1 < S.j1) {
                // average over the children that exist: 4, 2 or 1 (adjoint: as if all did)
                const float sc = (r < S.n1 || adjoint ? 0.5f : 1.f) * (oin || adjoint ? 0.5f : 1.f);
                const long long cc = (long long) (r >> 1) * cn0 + (S.ge >> 1);
                bc[cc] = __fmul_rn(__fadd_rn(__fadd_rn(pa, re), ro), sc);
                xc[cc] = 0.f;
            }
        } else {
            // full weighting about row r - 1 when it holds coarse nodes (the lane's even column does)
            const int rc = r - 1;
            if (((L.lo[1] + rc) & 1) == 0) {
                const float l2 = __shfl_up_sync(FULL, q2o, 1), l1 = __shfl_up_sync(FULL, q1o, 1), l0 = __shfl_up_sync(FULL, ro, 1);
                float acc = __fmaf_rn(0.0625f, l2, 0.f);
                acc = __fmaf_rn(0.125f, q2e, acc);
                acc = __fmaf_rn(0.0625f, q2o, acc);
                acc = __fmaf_rn(0.125f, l1, acc);
                acc = __fmaf_rn(0.25f, q1e, acc);
                acc = __fmaf_rn(0.125f, q1o, acc);
                acc = __fmaf_rn(0.0625f, l0, acc);
                acc = __fmaf_rn(0.125f, re, acc);
                acc = __fmaf_rn(0.0625f, ro, acc);
                const int I0 = ((L.lo[0] + S.ge) >> 1) - Lc.lo[0], I1 = ((L.lo[1] + rc) >> 1) - Lc.lo[1];
                if (own_e && rc >= S.j0 && rc < S.j1 && (unsigned) I0 < (unsigned) cn0 && (unsigned) I1 < (unsigned) Lc.n[1]) {
                    const long long cc = (long long) I1 * cn0 + I0;
                    bc[cc] = acc;
                    xc[cc] = 0.f;
                }
            }
            q2e = q1e;
            q2o = q1o;
            q1e = re;
            q1o = ro;
        }
    };
#pragma unroll
    for (int q = 0; q < PF; ++q) load(S.jb + q, B[LAG + q]);
#pragma unroll 1
    for (int jp = S.jb; jp <= S.je; jp += 2) {
        load(jp + PF, B[LAG + PF]);
        load(jp + PF + 1, B[LAG + PF + 1]);
        row(Par<0>{}, jp);
        row(Par<1>{}, jp + 1);
#pragma unroll
        for (int k = 0; k + 2 < NX; ++k) {
            X[k][0] = X[k + 2][0];
            X[k][1] = X[k + 2][1];
        }
#pragma unroll
        for (int k = 0; k + 2 < NB; ++k) {
            B[k][0] = B[k + 2][0];
            B[k][1] = B[k + 2][1];
        }
    }
}

// Index of a coarse row or column for interpolation by the boundary ghost rules, and the factor of its
// value: cell-centred levels mirror with the opposite sign at a GH_ZERO side, node-centred ones take 0
// there.  wrap: I may lie more than a period outside.
template <bool NODE>
__device__ __forceinline__ int ghost_pos(int I, int n, int lo_rule, int hi_rule, float& f, bool wrap = true) {
    f = 1.f;
    if ((unsigned) I < (unsigned) n) return I;
    const int rule = I < 0 ? lo_rule : hi_rule;
    if (rule == GH_WRAP) return wrap ? wrap_pos(I, n) : (I < 0 ? I + n : I - n);
    if (rule == GH_ZERO) f = NODE ? 0.f : -1.f;
    return I < 0 ? 0 : n - 1;
}

// Up-leg step: x = (pre-smoothed x) + P x_coarse, then SW red-black sweeps (colour 1 first).  The windows
// hold rows jp - LAG - 1 .. jp + 1 + PF of x and jp - LAG .. jp + 1 + PF of b (the last PF on their way).
template <int SW, bool NODE, int MODE>
__device__ __forceinline__ void strip_up(const LvlDev& L, const LvlDev& Lc, const Strip& S, int lane) {
    constexpr int LAG = 2 * SW;  // the last half sweep's row lags the newest row by this
    constexpr int NX = LAG + 3 + PF, NB = LAG + 2 + PF;
    const Column Ke = column_of<MODE>(S.te), Ko = column_of<MODE>(S.to);
    constexpr bool YIN = MODE == ROWS_INNER;
    const float* bg = L.b32;
    const float* xr = L.r32;
    float* xg = L.x32;
    const float* xc = Lc.x32;
    const int nc0 = Lc.n[0], nc1 = Lc.n[1];
    const bool own_e = S.ge >= S.i0 && S.ge < S.i1, own_o = S.ge + 1 >= S.i0 && S.ge + 1 < S.i1;
    // the lane's coarse column (of its even column), and the one beyond the warp that lanes 0 and 31 need
    const int I0 = NODE ? ((L.lo[0] + S.ist) >> 1) - Lc.lo[0] + lane : (S.ist >> 1) + lane;
    float fm, fe;
    const int cm = ghost_pos<NODE>(I0, nc0, Lc.gh_lo[0], Lc.gh_hi[0], fm);
    const int ce = ghost_pos<NODE>(lane == 0 ? I0 - 1 : I0 + 1, nc0, Lc.gh_lo[0], Lc.gh_hi[0], fe);
    float X[NX][2], B[NB][2];
#pragma unroll
    for (int k = 0; k < NX; ++k) X[k][0] = X[k][1] = 0.f;
#pragma unroll
    for (int k = 0; k < NB; ++k) B[k][0] = B[k][1] = 0.f;
    auto load = [&](int r, float (&xv)[2], float (&bv)[2]) {
        const bool ok = YIN || S.row_ok(r);
        const long long o = (long long) (YIN ? r : (ok ? S.row_of(r) : 0)) * S.n0;
        xv[0] = ok && S.oke ? ldf(xr + o + S.we) : 0.f;
        xv[1] = ok && S.oko ? ldf(xr + o + S.wo) : 0.f;
        bv[0] = ok && S.oke ? ldf(bg + o + S.we) : 0.f;
        bv[1] = ok && S.oko ? ldf(bg + o + S.wo) : 0.f;
    };
    // a coarse row as (left, own, right) columns; its raw part (own, edge) is loaded two fine rows ahead
    struct Raw { float m, e; };
    struct Row { float l, m, r; };
    auto craw = [&](int I) -> Raw {
        float f;
        const int ri = ghost_pos<NODE>(I, nc1, Lc.gh_lo[1], Lc.gh_hi[1], f, false);
        const float* p = xc + (long long) ri * nc0;
        Raw v;
        v.m = __fmul_rn(fm * f, ldf(p + cm));
        v.e = !NODE && (lane == 0 || lane == 31) ? __fmul_rn(fe * f, ldf(p + ce)) : 0.f;
        return v;
    };
    auto crow = [&](const Raw& v) -> Row {
        Row r;
        r.m = v.m;
        r.r = __shfl_down_sync(FULL, v.m, 1);
        r.l = 0.f;
        if (!NODE) {
            r.l = __shfl_up_sync(FULL, v.m, 1);
            if (lane == 0) r.l = v.e;
            if (lane == 31) r.r = v.e;
        }
        return r;
    };
    // Cell-centred (jb even): row 2 I interpolates coarse rows I, I - 1 (cc, cp), row 2 I + 1 rows I, I + 1
    // (cc, cn).  Node-centred: a row at an even node g takes coarse row g / 2 (cc), one at an odd node
    // (g - 1) / 2 and (g + 1) / 2 (cc, cn).  Before an even row the rows advance by one.
    const int g0 = L.lo[1] + S.jb;
    const int A0 = NODE ? (g0 >> 1) - Lc.lo[1] : (S.jb >> 1);
    const int odd0 = NODE ? (g0 & 1) : 0;  // 1: row jb is at an odd node
    Row cp = {0.f, 0.f, 0.f}, cc = crow(craw(A0 - 1 + odd0)), cn = crow(craw(A0 + odd0));
    Raw nx = craw(A0 + 1 + odd0);
    int In = A0 + 2 + odd0;  // the coarse row to load next
    auto row = [&](auto par, int j) {
        constexpr int P = decltype(par)::value;
        constexpr int kx = LAG + 1 + P, kb = LAG + P;
        const bool even = NODE ? (P ^ odd0) == 0 : P == 0;
        if (even) {
            cp = cc;
            cc = cn;
            cn = crow(nx);
            nx = craw(In++);
        }
        float ae, ao;
        if (!NODE) {
            const Row& o = P == 0 ? cp : cn;
            ae = __fmaf_rn(0.5625f, cc.m, 0.f);
            ae = __fmaf_rn(0.1875f, cc.l, ae);
            ae = __fmaf_rn(0.1875f, o.m, ae);
            ae = __fmaf_rn(0.0625f, o.l, ae);
            ao = __fmaf_rn(0.5625f, cc.m, 0.f);
            ao = __fmaf_rn(0.1875f, cc.r, ao);
            ao = __fmaf_rn(0.1875f, o.m, ao);
            ao = __fmaf_rn(0.0625f, o.r, ao);
        } else if (even) {
            ae = cc.m;
            ao = __fmaf_rn(0.5f, cc.r, __fmaf_rn(0.5f, cc.m, 0.f));
        } else {
            ae = __fmaf_rn(0.5f, cn.m, __fmaf_rn(0.5f, cc.m, 0.f));
            ao = __fmaf_rn(0.25f, cc.m, 0.f);
            ao = __fmaf_rn(0.25f, cc.r, ao);
            ao = __fmaf_rn(0.25f, cn.m, ao);
            ao = __fmaf_rn(0.25f, cn.r, ao);
        }
        // (columns and rows outside the level keep x = 0)
        const bool ok = YIN || S.row_ok(j);
        X[kx][0] = __fadd_rn(X[kx][0], ok && S.oke ? ae : 0.f);
        X[kx][1] = __fadd_rn(X[kx][1], ok && S.oko ? ao : 0.f);
        // half sweep h (colour h & 1) of row j - h
#pragma unroll
        for (int h = 1; h <= LAG; ++h) strip_gs<P, MODE>(S, j - h, X, kx - h, B[kb - h][P], Ke, Ko);
        const int r = j - LAG;
        if (r >= S.j0 && r < S.j1) {
            float* p = xg + (long long) r * S.n0 + S.ge;
            if (own_e) p[0] = X[kx - LAG][0];
            if (own_o) p[1] = X[kx - LAG][1];
        }
    };
#pragma unroll
    for (int q = 0; q < PF; ++q) load(S.jb + q, X[LAG + 1 + q], B[LAG + q]);
#pragma unroll 1
    for (int jp = S.jb; jp <= S.je; jp += 2) {
        load(jp + PF, X[LAG + 1 + PF], B[LAG + PF]);
        load(jp + PF + 1, X[LAG + 2 + PF], B[LAG + PF + 1]);
        row(Par<0>{}, jp);
        row(Par<1>{}, jp + 1);
#pragma unroll
        for (int k = 0; k + 2 < NX; ++k) {
            X[k][0] = X[k + 2][0];
            X[k][1] = X[k + 2][1];
        }
#pragma unroll
        for (int k = 0; k + 2 < NB; ++k) {
            B[k][0] = B[k + 2][0];
            B[k][1] = B[k + 2][1];
        }
    }
}

template <int SW, bool DOWN, int MODE>
__device__ __forceinline__ void strip_step(const LvlDev& L, const LvlDev& Lc, const Strip& S, int lane) {
    if constexpr (DOWN) Lc.node ? strip_down<SW, true, MODE>(L, Lc, S, lane) : strip_down<SW, false, MODE>(L, Lc, S, lane);
    else Lc.node ? strip_up<SW, true, MODE>(L, Lc, S, lane) : strip_up<SW, false, MODE>(L, Lc, S, lane);
}

// hxy: the halo the strips were cut for, 2 x (the larger of the two sweep counts), one more for levels
// with a node-centred coarse level
template <int SW, bool DOWN>
__global__ void __launch_bounds__(32 * STRIP_WARPS) mg_strip(const LvlDev* __restrict__ Ls, const Chunk* __restrict__ strips, int nstrips,
                                                            const Scal* sc, int hxy) {
    const int t = blockIdx.x * STRIP_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (t >= nstrips) return;  // (a whole warp)
    const Chunk C = strips[t];
    const LvlDev& L = Ls[C.lvl];
    if (sc && !sc[L.problem].active) return;
    const LvlDev& Lc = Ls[L.coarse];
    const bool node = Lc.node;
    const Strip S = strip_of(L, C, hxy + (node ? 1 : 0), 2 * SW + (DOWN && node ? 1 : 0), lane);
    // (the march runs in pairs of rows and loads PF rows past the last one)
    const int mode = S.jb >= 1 && S.je + PF + 2 <= S.n1 - 2 ? ROWS_INNER : (L.uoff ? ROWS_DIAG : ROWS_GENERAL);
    if (mode == ROWS_INNER) strip_step<SW, DOWN, ROWS_INNER>(L, Lc, S, lane);
    else if (mode == ROWS_DIAG) strip_step<SW, DOWN, ROWS_DIAG>(L, Lc, S, lane);
    else strip_step<SW, DOWN, ROWS_GENERAL>(L, Lc, S, lane);
}

bool mg_tiles_supported(int sweeps) { return sweeps >= 1 && sweeps <= MG_STRIP_SWEEPS; }

// Strips of level li with `rows` rows each: 64 columns less the halo on both sides.  A node-centred
// level's first strip starts where its even columns fall on coarse nodes.
void mg_strips(int li, const LvlDev& D, bool coarse_node, int sweeps, int rows, std::vector<Chunk>& out) {
    const int hx = 2 * sweeps + (coarse_node ? 1 : 0), w = 64 - 2 * hx;
    const int first = coarse_node && ((D.lo[0] - hx) & 1) ? -1 : 0;
    for (int j0 = 0; j0 < D.n[1]; j0 += rows)
        for (int i0 = first; i0 < D.n[0]; i0 += w) {
            Chunk c{li, j0, 0, i0, w};
            c.nrows = rows;
            out.push_back(c);
        }
}

template <bool DOWN>
static int launch_strips(cudaStream_t s, const LvlDev* L, const Chunk* strips, int n, const Scal* sc, int sweeps, int hxy, const char* name) {
    if (n <= 0) return OPFLOW_OK;
    const int g = (n + STRIP_WARPS - 1) / STRIP_WARPS;
    switch (sweeps) {
        case 1: mg_strip<1, DOWN><<<g, 32 * STRIP_WARPS, 0, s>>>(L, strips, n, sc, hxy); break;
        case 2: mg_strip<2, DOWN><<<g, 32 * STRIP_WARPS, 0, s>>>(L, strips, n, sc, hxy); break;
        case 3: mg_strip<3, DOWN><<<g, 32 * STRIP_WARPS, 0, s>>>(L, strips, n, sc, hxy); break;
        case 4: mg_strip<4, DOWN><<<g, 32 * STRIP_WARPS, 0, s>>>(L, strips, n, sc, hxy); break;
        default: return fail(OPFLOW_E_INVALID, "%s: %d sweeps", name, sweeps);
    }
    OPG_LAUNCHED();
    return check_launch(name);
}

int mg_launch_tile_down(cudaStream_t s, const LvlDev* L, const Chunk* strips, int n, const Scal* sc, int pre, int post) {
    return launch_strips<true>(s, L, strips, n, sc, pre, 2 * std::max(pre, post), "mg_strip (down)");
}

int mg_launch_tile_up(cudaStream_t s, const LvlDev* L, const Chunk* strips, int n, const Scal* sc, int pre, int post) {
    return launch_strips<false>(s, L, strips, n, sc, post, 2 * std::max(pre, post), "mg_strip (up)");
}

}  // namespace opg
