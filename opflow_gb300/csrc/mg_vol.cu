// Fused 3D multigrid steps of the red-black float32 levels with a class-table operator: the 3D form of
// mg_tiles.cu.  A CTA takes a 64 x 32 patch of the xy plane and marches it along z through the whole
// down-leg step - pre-smoothing from a zero guess, residual, restriction - or the whole up-leg step -
// prolongation, post-smoothing.
//
//  - A warp holds two rows of 64 columns, lane l the columns 2l and 2l + 1 of both, a window of planes of
//    them in registers.  On every plane a half sweep updates one cell of each row and lane; the
//    x-neighbours come by shuffle, the z-neighbours and one y-neighbour from the thread's own registers.
//  - Half sweep h works one plane behind half sweep h - 1 and the residual one plane behind the last, so
//    a step of the march takes one new plane through the whole pipeline.  A stage reads, of its own plane,
//    only what the stage before it left there one step earlier: the y-neighbours in the adjacent warps'
//    rows are published in shared memory at the end of each step (two buffers), one barrier per step.
//  - Every half sweep invalidates one more cell at the patch's edge: of 64 x 32 x (planes + 8) cells the
//    inner 56 x 24 x planes are the CTA's own (two sweeps).
// Level data crosses memory once per step (down: b in, x and coarse b out; up: x, b, coarse x in, x out)
// instead of once per half sweep, residual, restriction and prolongation.  The per-cell arithmetic is the
// chunked kernels' in their operation order, so the iterates are theirs bit for bit.  As in mg_tiles.cu
// the launch never writes what it reads: the smoothed x of the down step lies in r until the up step.
//
// Levels: cell-centred, not periodic, off-diagonal coefficients the interior class's everywhere
// (LvlDev::uoff: the classes differ in the centre coefficient only); a cell outside the level has an inverse
// diagonal of 0, so its x stays 0, the value that makes an absent neighbour's term vanish.
//
// What bounds it: instruction issue (0.6 / 0.5 of the slots; 199 / 334 warp instructions per plane of a
// warp's 128 cells, 65 % of which are its own) and, with one CTA per SM, the barrier per plane.  256^3
// level, down: 81 us against 290 for four half sweeps, residual and restriction; up: 153 us against 230 for
// prolongation and four half sweeps.  Levels below 64^3: 14 to 20 us per leg, against 5 to 10 us for
// each of eleven launches.  256^3 mixed solve 14.0 -> 10.1 ms.
#include "mg_device.h"

#include <type_traits>

namespace opg {

constexpr int VOL_WARPS = 16, VOL_ROWS = 2 * VOL_WARPS;
constexpr unsigned VFULL = 0xffffffffu;
constexpr int VOL_PF = 2;  // planes of loads in flight ahead of the march

// the y-edges of a warp's two rows, published for the adjacent warps: [buffer][plane of the pipeline][warp][row]
template <int NPUB>
struct VolShared {
    float edge[2][NPUB][VOL_WARPS][2][32];
    float c0[28], inv[28];  // per class; 27: outside the level
};

struct VolTile {
    int n0, n1, n2;
    int ist, y0;          // lane 0's even column, the warp's first row
    int jb, je;           // first and last plane the march needs (it runs in pairs of planes from jb)
    int k0, k1;           // the CTA's own planes
    int i1, j1;           // its own columns end before i1, rows before j1 (they start at ist + hx, ...)
    int i0, j0;
    int ge;               // the lane's even column
    bool oke, oko, okr[2];
    int cls[2][2];        // class of (row, column) in an inner plane's numbering (x + 3 y), -1 outside
};

// the cell's class index in plane p, 27 outside the level
__device__ __forceinline__ int vol_class(const VolTile& T, int r, int c, int p) {
    const int z = p == 0 ? 0 : (p == T.n2 - 1 ? 18 : 9);
    return T.cls[r][c] < 0 || (unsigned) p >= (unsigned) T.n2 ? 27 : T.cls[r][c] + z;
}

// the off-diagonal coefficients, and of the thread's four cells the centre one and its inverse on planes
// away from the level's first and last
struct VolCoef {
    float cx0, cx1, cy0, cy1, cz0, cz1;
    float c0[2][2], inv[2][2];
};

// off-diagonal sum of the cell (column P) of a row: W and E from the row's other column
template <int P>
__device__ __forceinline__ float vol_offdiag(const VolCoef& K, const float (&row)[2], float s, float n, float d, float u) {
    const float w = P == 0 ? __shfl_up_sync(VFULL, row[1], 1) : row[0];
    const float e = P == 0 ? row[1] : __shfl_down_sync(VFULL, row[0], 1);
    float acc = __fmaf_rn(K.cx0, w, 0.f);
    acc = __fmaf_rn(K.cx1, e, acc);
    acc = __fmaf_rn(K.cy0, s, acc);
    acc = __fmaf_rn(K.cy1, n, acc);
    acc = __fmaf_rn(K.cz0, d, acc);
    return __fmaf_rn(K.cz1, u, acc);
}

template <int P>
struct VPar {
    static constexpr int value = P;
};

__device__ __forceinline__ VolTile vol_tile(const LvlDev& L, const Chunk& C, int h) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    VolTile T;
    T.n0 = L.n[0];
    T.n1 = L.n[1];
    T.n2 = L.n[2];
    T.i0 = C.i0;
    T.j0 = C.j;
    T.k0 = C.k;
    T.i1 = min(C.i0 + 64 - 2 * h, T.n0);
    T.j1 = min(C.j + VOL_ROWS - 2 * h, T.n1);
    T.k1 = min(C.k + C.nrows, T.n2);
    T.ist = C.i0 - h;
    T.y0 = C.j - h + 2 * warp;
    T.jb = C.k - h;  // (even, as ist and y0: a cell's colour is that of its column, row and plane parities)
    T.je = min(C.k + C.nrows, (T.n2 + 1) & ~1) - 1 + h;
    T.ge = T.ist + 2 * lane;
    T.oke = (unsigned) T.ge < (unsigned) T.n0;
    T.oko = (unsigned) (T.ge + 1) < (unsigned) T.n0;
    for (int r = 0; r < 2; ++r) {
        const int y = T.y0 + r;
        T.okr[r] = (unsigned) y < (unsigned) T.n1;
        T.cls[r][0] = T.okr[r] && T.oke ? pos_class(T.ge, T.n0) + 3 * pos_class(y, T.n1) : -1;
        T.cls[r][1] = T.okr[r] && T.oko ? pos_class(T.ge + 1, T.n0) + 3 * pos_class(y, T.n1) : -1;
    }
    return T;
}

// fills the class tables' centre coefficients and inverses (a barrier before their first use follows)
template <typename SH>
__device__ __forceinline__ void vol_tables(const LvlDev& L, SH& sh) {
    for (int q = threadIdx.x; q < 28; q += blockDim.x) {
        sh.c0[q] = q < NCLASS ? L.T32[q * TSTRIDE] : 0.f;
        sh.inv[q] = q < NCLASS ? L.T32[q * TSTRIDE + NSLOT] : 0.f;
    }
}
template <typename SH>
__device__ __forceinline__ VolCoef vol_coefs(const LvlDev& L, const VolTile& T, const SH& sh) {
    const float* t = L.T32 + 13 * TSTRIDE;
    VolCoef K{t[1], t[2], t[3], t[4], t[5], t[6]};
    for (int r = 0; r < 2; ++r)
        for (int c = 0; c < 2; ++c) {
            const int q = T.cls[r][c] < 0 ? 27 : T.cls[r][c] + 9;
            K.c0[r][c] = sh.c0[q];
            K.inv[r][c] = sh.inv[q];
        }
    return K;
}

// SW sweeps from x = 0, residual, restriction.  The windows hold planes jp - LAG - 1 .. jp + 1 of x and
// jp - LAG .. jp + 1 + VOL_PF of b for the pair of planes (jp, jp + 1).
template <int SW, typename SH>
__device__ __forceinline__ void vol_down(const LvlDev& L, const LvlDev& Lc, const VolTile& T, const VolCoef& K, SH& sh) {
    constexpr int LAG = 2 * SW, NX = LAG + 3, NB = LAG + 2 + VOL_PF;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wd = max(warp - 1, 0), wu = min(warp + 1, VOL_WARPS - 1);  // (beyond the patch: any finite value)
    const long long sy = T.n0, sz = (long long) T.n0 * T.n1;
    const float* bg = L.b32 + T.ge + sy * T.y0;
    float* xg = L.r32 + T.ge + sy * T.y0;
    const bool adjoint = L.adjoint;
    const bool own_e = T.ge >= T.i0 && T.ge < T.i1, own_o = T.ge + 1 >= T.i0 && T.ge + 1 < T.i1;
    bool own_r[2];
    for (int r = 0; r < 2; ++r) own_r[r] = T.y0 + r >= T.j0 && T.y0 + r < T.j1;
    float X[NX][2][2], B[NB][2][2];
#pragma unroll
    for (int k = 0; k < NX; ++k) X[k][0][0] = X[k][0][1] = X[k][1][0] = X[k][1][1] = 0.f;
#pragma unroll
    for (int k = 0; k < NB; ++k) B[k][0][0] = B[k][0][1] = B[k][1][0] = B[k][1][1] = 0.f;
    auto load = [&](int p, float (&v)[2][2]) {
        const bool okp = (unsigned) p < (unsigned) T.n2;
        const float* q = bg + sz * p;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            v[r][0] = okp && T.okr[r] && T.oke ? __ldg(q + r * sy) : 0.f;
            v[r][1] = okp && T.okr[r] && T.oko ? __ldg(q + r * sy + 1) : 0.f;
        }
    };
    float pa = 0.f;  // the even plane's part of the coarse sum
    // ZIN: every plane of the pipeline is inside the level, away from its first and last one
    auto plane = [&](auto par, auto zin, int j, int buf) {
        constexpr bool ZIN = decltype(zin)::value;
        auto inv_of = [&](int r, int c, int p) { return ZIN ? K.inv[r][c] : sh.inv[vol_class(T, r, c, p)]; };
        auto c0_of = [&](int r, int c, int p) { return ZIN ? K.c0[r][c] : sh.c0[vol_class(T, r, c, p)]; };
        constexpr int U = decltype(par)::value;             // plane j = jp + U
        constexpr int kx = LAG + 1 + U, kb = LAG + U;       // plane j in X and B
        constexpr int P0 = U, P1 = 1 - U;                   // the column every stage of this step updates in row 0 and 1
        // half sweep 1 (colour 0) from the zero guess
        X[kx][0][P1] = X[kx][1][P0] = 0.f;
        X[kx][0][P0] = __fmul_rn(B[kb][0][P0], inv_of(0, P0, j));
        X[kx][1][P1] = __fmul_rn(B[kb][1][P1], inv_of(1, P1, j));
        // half sweep d + 1 of plane j - d
#pragma unroll
        for (int d = 1; d < LAG; ++d) {
            const int k = kx - d, p = j - d;
            const float south = sh.edge[buf][d - 1][wd][1][lane], north = sh.edge[buf][d - 1][wu][0][lane];
            const float a0 = vol_offdiag<P0>(K, X[k][0], south, X[k][1][P0], X[k - 1][0][P0], X[k + 1][0][P0]);
            const float a1 = vol_offdiag<P1>(K, X[k][1], X[k][0][P1], north, X[k - 1][1][P1], X[k + 1][1][P1]);
            const float v0 = __fmul_rn(__fsub_rn(B[kb - d][0][P0], a0), inv_of(0, P0, p));
            const float v1 = __fmul_rn(__fsub_rn(B[kb - d][1][P1], a1), inv_of(1, P1, p));
            X[k][0][P0] = v0;
            X[k][1][P1] = v1;
        }
        // the residual of plane p, whose x is final
        const int p = j - LAG;
        constexpr int k = kx - LAG;
        float res[2][2];
        {
            const float* es = sh.edge[buf][LAG - 1][wd][1];
            const float* en = sh.edge[buf][LAG - 1][wu][0];
            const float* es2 = sh.edge[buf][LAG][wd][1];
            const float* en2 = sh.edge[buf][LAG][wu][0];
            float a[2][2];
            a[0][P0] = vol_offdiag<P0>(K, X[k][0], es[lane], X[k][1][P0], X[k - 1][0][P0], X[k + 1][0][P0]);
            a[0][P1] = vol_offdiag<P1>(K, X[k][0], es2[lane], X[k][1][P1], X[k - 1][0][P1], X[k + 1][0][P1]);
            a[1][P1] = vol_offdiag<P1>(K, X[k][1], X[k][0][P1], en[lane], X[k - 1][1][P1], X[k + 1][1][P1]);
            a[1][P0] = vol_offdiag<P0>(K, X[k][1], X[k][0][P0], en2[lane], X[k - 1][1][P0], X[k + 1][1][P0]);
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    res[r][c] = __fsub_rn(B[kb - LAG][r][c], __fmaf_rn(c0_of(r, c, p), X[k][r][c], a[r][c]));
                    if (!T.okr[r] || !(c ? T.oko : T.oke) || (!ZIN && (unsigned) p >= (unsigned) T.n2)) res[r][c] = 0.f;
                }
        }
        if (p >= T.k0 && p < T.k1) {
            float* q = xg + sz * p;
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                if (own_r[r] && own_e) q[r * sy] = X[k][r][0];
                if (own_r[r] && own_o) q[r * sy + 1] = X[k][r][1];
            }
        }
        // (jb, y0 and the even column are even: planes, rows and columns 2 I, 2 I + 1 come in pairs)
        if (U == 0) {
            pa = __fadd_rn(__fadd_rn(__fadd_rn(res[0][0], res[0][1]), res[1][0]), res[1][1]);
        } else {
            const float acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(pa, res[0][0]), res[0][1]), res[1][0]), res[1][1]);
            if (own_e && own_r[0] && p - 1 >= T.k0 && p - 1 < T.k1) {
                // average over the children that exist: 8, 4, 2 or 1 (adjoint: as if all did)
                const float sc = adjoint ? 0.125f : (p < T.n2 ? 0.5f : 1.f) * (T.okr[1] ? 0.5f : 1.f) * (T.oko ? 0.5f : 1.f);
                const long long cc = (T.ge >> 1) + (long long) Lc.n[0] * ((T.y0 >> 1) + (long long) Lc.n[1] * (p >> 1));
                Lc.b32[cc] = __fmul_rn(acc, sc);
                Lc.x32[cc] = 0.f;
            }
        }
        // the next step's stages: plane j - d of what is now plane j - (d - 1), the column they read of a
        // neighbouring row (row 1 for the warp above: its row 0 updates column P1; row 0 for the one below)
#pragma unroll
        for (int d = 1; d < LAG; ++d) {
            sh.edge[buf ^ 1][d - 1][warp][1][lane] = X[kx - (d - 1)][1][P1];
            sh.edge[buf ^ 1][d - 1][warp][0][lane] = X[kx - (d - 1)][0][P0];
        }
        sh.edge[buf ^ 1][LAG - 1][warp][1][lane] = X[kx - (LAG - 1)][1][P1];
        sh.edge[buf ^ 1][LAG - 1][warp][0][lane] = X[kx - (LAG - 1)][0][P0];
        sh.edge[buf ^ 1][LAG][warp][1][lane] = X[kx - (LAG - 1)][1][P0];
        sh.edge[buf ^ 1][LAG][warp][0][lane] = X[kx - (LAG - 1)][0][P1];
        __syncthreads();
    };
#pragma unroll
    for (int q = 0; q < VOL_PF; ++q) load(T.jb + q, B[LAG + q]);
#pragma unroll 1
    for (int jp = T.jb; jp <= T.je; jp += 2) {
        load(jp + VOL_PF, B[LAG + VOL_PF]);
        load(jp + VOL_PF + 1, B[LAG + VOL_PF + 1]);
        if (jp - LAG >= 1 && jp + 1 <= T.n2 - 2) {
            plane(VPar<0>{}, std::true_type{}, jp, 0);
            plane(VPar<1>{}, std::true_type{}, jp + 1, 1);
        } else {
            plane(VPar<0>{}, std::false_type{}, jp, 0);
            plane(VPar<1>{}, std::false_type{}, jp + 1, 1);
        }
#pragma unroll
        for (int k = 0; k + 2 < NX; ++k)
#pragma unroll
            for (int q = 0; q < 4; ++q) X[k][q >> 1][q & 1] = X[k + 2][q >> 1][q & 1];
#pragma unroll
        for (int k = 0; k + 2 < NB; ++k)
#pragma unroll
            for (int q = 0; q < 4; ++q) B[k][q >> 1][q & 1] = B[k + 2][q >> 1][q & 1];
    }
}

// index of a coarse cell along one dim by the boundary ghost rules, and the factor of its value
__device__ __forceinline__ int vol_ghost(int I, int n, int lo_rule, int hi_rule, float& f) {
    f = 1.f;
    if ((unsigned) I < (unsigned) n) return I;
    if ((I < 0 ? lo_rule : hi_rule) == GH_ZERO) f = -1.f;
    return I < 0 ? 0 : n - 1;
}

// x = (pre-smoothed x) + P x_coarse, SW sweeps (colour 1 first).  The windows hold planes
// jp - LAG - 1 .. jp + 1 + VOL_PF of x and jp - LAG .. jp + 1 + VOL_PF of b.
template <int SW, typename SH>
__device__ __forceinline__ void vol_up(const LvlDev& L, const LvlDev& Lc, const VolTile& T, const VolCoef& K, SH& sh) {
    constexpr int LAG = 2 * SW, NX = LAG + 3 + VOL_PF, NB = LAG + 2 + VOL_PF;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wd = max(warp - 1, 0), wu = min(warp + 1, VOL_WARPS - 1);
    const long long sy = T.n0, sz = (long long) T.n0 * T.n1;
    const float* bg = L.b32 + T.ge + sy * T.y0;
    const float* xr = L.r32 + T.ge + sy * T.y0;
    float* xg = L.x32 + T.ge + sy * T.y0;
    const float* xc = Lc.x32;
    const bool own_e = T.ge >= T.i0 && T.ge < T.i1, own_o = T.ge + 1 >= T.i0 && T.ge + 1 < T.i1;
    bool own_r[2];
    for (int r = 0; r < 2; ++r) own_r[r] = T.y0 + r >= T.j0 && T.y0 + r < T.j1;
    // the coarse cells: the lane's column and the one beyond the warp that lanes 0 and 31 need, three rows
    const int nc0 = Lc.n[0], nc1 = Lc.n[1], nc2 = Lc.n[2];
    const int I0 = (T.ist >> 1) + lane;
    float fm, fe, fr[3];
    const int cm = vol_ghost(I0, nc0, Lc.gh_lo[0], Lc.gh_hi[0], fm);
    const int ce = vol_ghost(lane == 0 ? I0 - 1 : I0 + 1, nc0, Lc.gh_lo[0], Lc.gh_hi[0], fe);
    int cr[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) cr[q] = vol_ghost((T.y0 >> 1) - 1 + q, nc1, Lc.gh_lo[1], Lc.gh_hi[1], fr[q]);
    const long long csz = (long long) nc0 * nc1;
    float X[NX][2][2], B[NB][2][2];
#pragma unroll
    for (int k = 0; k < NX; ++k) X[k][0][0] = X[k][0][1] = X[k][1][0] = X[k][1][1] = 0.f;
#pragma unroll
    for (int k = 0; k < NB; ++k) B[k][0][0] = B[k][0][1] = B[k][1][0] = B[k][1][1] = 0.f;
    auto load = [&](int p, float (&xv)[2][2], float (&bv)[2][2]) {
        const bool okp = (unsigned) p < (unsigned) T.n2;
        const float *q = bg + sz * p, *s = xr + sz * p;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const bool e = okp && T.okr[r] && T.oke, o = okp && T.okr[r] && T.oko;
            bv[r][0] = e ? __ldg(q + r * sy) : 0.f;
            bv[r][1] = o ? __ldg(q + r * sy + 1) : 0.f;
            xv[r][0] = e ? __ldg(s + r * sy) : 0.f;
            xv[r][1] = o ? __ldg(s + r * sy + 1) : 0.f;
        }
    };
    // a coarse plane: three rows of (left, own, right); its raw part is loaded two fine planes ahead
    struct Raw { float m[3], e[3]; };
    struct Pl { float v[3][3]; };
    auto craw = [&](int Kp) -> Raw {
        float f;
        const float* p = xc + csz * vol_ghost(Kp, nc2, Lc.gh_lo[2], Lc.gh_hi[2], f);
        Raw a;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            a.m[q] = __fmul_rn(fm * fr[q] * f, __ldg(p + (long long) cr[q] * nc0 + cm));
            a.e[q] = lane == 0 || lane == 31 ? __fmul_rn(fe * fr[q] * f, __ldg(p + (long long) cr[q] * nc0 + ce)) : 0.f;
        }
        return a;
    };
    auto cplane = [&](const Raw& a) -> Pl {
        Pl c;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            c.v[q][1] = a.m[q];
            c.v[q][0] = __shfl_up_sync(VFULL, a.m[q], 1);
            c.v[q][2] = __shfl_down_sync(VFULL, a.m[q], 1);
            if (lane == 0) c.v[q][0] = a.e[q];
            if (lane == 31) c.v[q][2] = a.e[q];
        }
        return c;
    };
    Pl cp, cc, cn;
    const int A0 = T.jb >> 1;
    cc = cplane(craw(A0 - 1));
    cn = cplane(craw(A0));
    Raw nx = craw(A0 + 1);
    int In = A0 + 2;
    auto plane = [&](auto par, auto zin, int j, int buf) {
        constexpr bool ZIN = decltype(zin)::value;
        auto inv_of = [&](int r, int c, int p) { return ZIN ? K.inv[r][c] : sh.inv[vol_class(T, r, c, p)]; };
        constexpr int U = decltype(par)::value;
        constexpr int kx = LAG + 1 + U, kb = LAG + U;
        constexpr int P0 = U, P1 = 1 - U;  // (half sweep h: plane j - h, colour h & 1)
        if (U == 0) {  // fine planes 2 I and 2 I + 1 take coarse planes I, I - 1 and I, I + 1
            cp = cc;
            cc = cn;
            cn = cplane(nx);
            nx = craw(In++);
        }
        const Pl& co = U == 0 ? cp : cn;
        const bool okp = ZIN || (unsigned) j < (unsigned) T.n2;
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                // row y0 + r takes coarse rows 1, 0 (r = 0) or 1, 2; column c coarse columns 1, 0 or 1, 2
                const int ry = r == 0 ? 0 : 2, cx = c == 0 ? 0 : 2;
                float a = __fmaf_rn(0.421875f, cc.v[1][1], 0.f);
                a = __fmaf_rn(0.140625f, cc.v[1][cx], a);
                a = __fmaf_rn(0.140625f, cc.v[ry][1], a);
                a = __fmaf_rn(0.046875f, cc.v[ry][cx], a);
                a = __fmaf_rn(0.140625f, co.v[1][1], a);
                a = __fmaf_rn(0.046875f, co.v[1][cx], a);
                a = __fmaf_rn(0.046875f, co.v[ry][1], a);
                a = __fmaf_rn(0.015625f, co.v[ry][cx], a);
                X[kx][r][c] = __fadd_rn(X[kx][r][c], okp && T.okr[r] && (c ? T.oko : T.oke) ? a : 0.f);
            }
#pragma unroll
        for (int h = 1; h <= LAG; ++h) {
            const int k = kx - h, p = j - h;
            const float south = sh.edge[buf][h - 1][wd][1][lane], north = sh.edge[buf][h - 1][wu][0][lane];
            const float a0 = vol_offdiag<P0>(K, X[k][0], south, X[k][1][P0], X[k - 1][0][P0], X[k + 1][0][P0]);
            const float a1 = vol_offdiag<P1>(K, X[k][1], X[k][0][P1], north, X[k - 1][1][P1], X[k + 1][1][P1]);
            const float v0 = __fmul_rn(__fsub_rn(B[kb - h][0][P0], a0), inv_of(0, P0, p));
            const float v1 = __fmul_rn(__fsub_rn(B[kb - h][1][P1], a1), inv_of(1, P1, p));
            X[k][0][P0] = v0;
            X[k][1][P1] = v1;
        }
        const int p = j - LAG;
        constexpr int k = kx - LAG;
        if (p >= T.k0 && p < T.k1) {
            float* q = xg + sz * p;
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                if (own_r[r] && own_e) q[r * sy] = X[k][r][0];
                if (own_r[r] && own_o) q[r * sy + 1] = X[k][r][1];
            }
        }
        // the next step's half sweep h: plane j - (h - 1), row 1's column its row-0 neighbour updates, row 0's
        // column its row-1 neighbour updates
#pragma unroll
        for (int h = 1; h <= LAG; ++h) {
            sh.edge[buf ^ 1][h - 1][warp][1][lane] = X[kx - (h - 1)][1][P1];
            sh.edge[buf ^ 1][h - 1][warp][0][lane] = X[kx - (h - 1)][0][P0];
        }
        __syncthreads();
    };
#pragma unroll
    for (int q = 0; q < VOL_PF; ++q) load(T.jb + q, X[LAG + 1 + q], B[LAG + q]);
#pragma unroll 1
    for (int jp = T.jb; jp <= T.je; jp += 2) {
        load(jp + VOL_PF, X[LAG + 1 + VOL_PF], B[LAG + VOL_PF]);
        load(jp + VOL_PF + 1, X[LAG + 2 + VOL_PF], B[LAG + VOL_PF + 1]);
        if (jp - LAG >= 1 && jp + 1 <= T.n2 - 2) {
            plane(VPar<0>{}, std::true_type{}, jp, 0);
            plane(VPar<1>{}, std::true_type{}, jp + 1, 1);
        } else {
            plane(VPar<0>{}, std::false_type{}, jp, 0);
            plane(VPar<1>{}, std::false_type{}, jp + 1, 1);
        }
#pragma unroll
        for (int k = 0; k + 2 < NX; ++k)
#pragma unroll
            for (int q = 0; q < 4; ++q) X[k][q >> 1][q & 1] = X[k + 2][q >> 1][q & 1];
#pragma unroll
        for (int k = 0; k + 2 < NB; ++k)
#pragma unroll
            for (int q = 0; q < 4; ++q) B[k][q >> 1][q & 1] = B[k + 2][q >> 1][q & 1];
    }
}

template <int SW, bool DOWN>
__global__ void __launch_bounds__(32 * VOL_WARPS, 1) mg_vol(const LvlDev* __restrict__ Ls, const Chunk* __restrict__ tiles, const Scal* sc) {
    __shared__ VolShared<2 * SW + 1> sh;
    const Chunk C = tiles[blockIdx.x];
    const LvlDev& L = Ls[C.lvl];
    if (sc && !sc[L.problem].active) return;  // (the whole CTA)
    const LvlDev& Lc = Ls[L.coarse];
    const VolTile T = vol_tile(L, C, 2 * SW);
    vol_tables(L, sh);
    {
        float* e = &sh.edge[0][0][0][0][0];
        for (int q = threadIdx.x; q < (int) (sizeof sh.edge / sizeof(float)); q += blockDim.x) e[q] = 0.f;
    }
    __syncthreads();
    const VolCoef K = vol_coefs(L, T, sh);
    if constexpr (DOWN) vol_down<SW>(L, Lc, T, K, sh);
    else vol_up<SW>(L, Lc, T, K, sh);
}

bool mg_vol_supported(int pre, int post) { return pre == post && pre >= 1 && pre <= 2; }

// Tiles of level li.  `choice` 4: the planes per tile (even) that minimise rounds of CTAs x (planes + halo);
// 2, 8, 16: half, two and four times as many (the tuner's alternatives).
void mg_vol_tiles(int li, const LvlDev& D, int sweeps, int sms, int choice, std::vector<Chunk>& out) {
    const int h = 2 * sweeps, w = 64 - 2 * h, rows = VOL_ROWS - 2 * h, all = (D.n[2] + 1) & ~1;
    const long long across = (long long) ((D.n[0] + w - 1) / w) * ((D.n[1] + rows - 1) / rows);
    int planes = 4;
    long long best = -1;
    for (int z = 4; z <= std::max(4, all); z += 2) {
        const long long rounds = (across * ((D.n[2] + z - 1) / z) + sms - 1) / sms, cost = rounds * (z + 2 * h + 2);
        if (best < 0 || cost < best) {
            best = cost;
            planes = z;
        }
    }
    planes = choice == 2 ? std::max(4, (planes / 2 + 1) & ~1) : std::min(std::max(4, all), choice == 8 ? 2 * planes : (choice == 16 ? 4 * planes : planes));
    for (int k0 = 0; k0 < D.n[2]; k0 += planes)
        for (int j0 = 0; j0 < D.n[1]; j0 += rows)
            for (int i0 = 0; i0 < D.n[0]; i0 += w) {
                Chunk c{li, j0, k0, i0, w};
                c.nrows = planes;
                out.push_back(c);
            }
}

int mg_launch_vol(cudaStream_t s, const LvlDev* L, const Chunk* tiles, int n, const Scal* sc, int sweeps, bool down) {
    if (n <= 0) return OPFLOW_OK;
    if (sweeps == 1 && down) mg_vol<1, true><<<n, 32 * VOL_WARPS, 0, s>>>(L, tiles, sc);
    else if (sweeps == 1) mg_vol<1, false><<<n, 32 * VOL_WARPS, 0, s>>>(L, tiles, sc);
    else if (sweeps == 2 && down) mg_vol<2, true><<<n, 32 * VOL_WARPS, 0, s>>>(L, tiles, sc);
    else if (sweeps == 2) mg_vol<2, false><<<n, 32 * VOL_WARPS, 0, s>>>(L, tiles, sc);
    else return fail(OPFLOW_E_INVALID, "mg_vol: %d sweeps", sweeps);
    OPG_LAUNCHED();
    return check_launch("mg_vol");
}

}  // namespace opg
