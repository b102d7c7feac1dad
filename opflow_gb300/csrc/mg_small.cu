// The V-cycle at and below a problem's first small level, one CTA per problem, with those levels' x and b in
// shared memory: float32 class-table levels whose classes differ in the centre coefficient only
// (LvlDev::uoff), red-black, 2D or 3D, cell- or node-centred, down to a coarsest level with a dense inverse.
//
// What bounds such levels is latency: a half sweep of a few thousand cells is a few passes of a CTA, each a
// chain of five shared-memory reads, five dependent operations and a barrier (about 200 cycles), where a
// launch or a strip's march over the level's rows takes microseconds.  So cells are spread over all threads,
// one barrier per half sweep among the warps that a level needs.  A thread forms its cells' places and inverse
// centres once for all half sweeps of a level, and the levels' geometry comes laid out by the host in one piece.  The
// code stays short (loops are not unrolled): a launch finds it cold in the instruction caches, and fetching an
// unrolled version took a third of the time.  Levels are framed by a ring of zeros, so that a neighbour that does not
// exist costs no test (its coefficient times 0 leaves the sum as it is).  A half sweep's warp takes 16 cells of one row and 16 of the
// next, whose colours alternate, so that its shared-memory accesses fall into distinct banks.
//
// The per-cell arithmetic is the chunked kernels' in their operation order (bit-identical iterates).  Measured,
// a level of 64^2 and all below it: 27 us, where strips take 20 us for that level alone and took 28 for the rest
// in one CTA; 16^3 and below 32 us, where the per-cell kernel took 45 for 8^3.
#include "mg_device.h"

#include <algorithm>
#include <cstring>

namespace opg {

constexpr int SM_THREADS = 1024, SM_WARPS = SM_THREADS / 32;
// q / d for q, d < 2^16, m = small_magic(d)
__device__ __forceinline__ int small_div(int q, unsigned m) { return m ? (int) __umulhi((unsigned) q, m) : q; }

// Barrier of the first `warps` warps.  Warps that a level does not need wait for the next larger one at that
// level's barrier meanwhile, so every level has its own (id: 1 + its index; all warps: the CTA's own).
__device__ __forceinline__ void small_sync(int warps, int id) {
    if (warps == SM_WARPS) __syncthreads();
    else if (warps == 1) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(warps * 32) : "memory");
}
static_assert(MG_BOTTOM_LEVELS <= 15, "a named barrier per level");

// One thread's part of a level.  Its places and inverse centres are indexed in loops that stay rolled, so they lie in
// local memory (64 bytes a thread, in the L1): read once per half sweep, ahead of the shared memory.  A warp share is 32 column pairs: 16 of two rows, or 8 of four or 4 of eight
// where the rows are short; a thread holds up to MG_SMALL_SHARES pairs (the cells of colour 0 and 1 next to each
// other).  A level of fewer shares than warps is run by the first `act` warps alone, the others go on to where
// the next larger level needs them again.
template <int ND, bool PER>
struct Small {
    const SmLevel& L;
    float* sm;
    int warp, lane, cnt;     // cnt: the thread's shares (the warp's, uniform)
    int act;                 // warps that run the level
    int s1, s2;
    float c[2 * ND];
    int o[MG_SMALL_SHARES];            // offset of the pair's even column
    int par;                           // bit q: the even column's colour in share q
    float inv[MG_SMALL_SHARES][2];     // 1 / centre of the even and the odd column, 0 where there is no cell

    __device__ __forceinline__ void sync() const { small_sync(act, L.barrier); }
    __device__ __forceinline__ void place(int q, int& t, int& j, int& k) const {
        const int g = warp + q * SM_WARPS, rp = small_div(g, L.mhalf);
        k = ND > 2 ? small_div(rp, L.mrows) : 0;
        j = ((rp - k * L.pairs) << (5 - L.lw)) + (lane >> L.lw);
        t = ((g - rp * L.half) << L.lw) + (lane & ((1 << L.lw) - 1));
    }
    __device__ __forceinline__ int cls(int i, int j, int k) const {
        return pos_class(i, L.n[0]) + 3 * pos_class(j, L.n[1]) + (ND > 2 ? 9 * pos_class(k, L.n[2]) : 0);
    }
    __device__ __forceinline__ Small(const SmLevel& l, float* s) : L(l), sm(s) {
        warp = threadIdx.x >> 5;
        lane = threadIdx.x & 31;
        act = min(L.shares, SM_WARPS);
        cnt = (L.shares - warp + SM_WARPS - 1) / SM_WARPS;
        s1 = L.s1;
        s2 = L.s2;
        par = 0;
#pragma unroll
        for (int q = 0; q < 2 * ND; ++q) c[q] = L.c[q];
#pragma unroll 1
        for (int q = 0; q < cnt; ++q) {
            o[q] = 0;
            inv[q][0] = inv[q][1] = 0.f;
            int t, j, k;
            place(q, t, j, k);
            const bool row = j < L.n[1];
            const int i = 2 * t;
            if (row && i < L.n[0]) {
                o[q] = i + j * s1 + (ND > 2 ? k * s2 : 0);
                inv[q][0] = L.inv[cls(i, j, k)];
                if (i + 1 < L.n[0]) inv[q][1] = L.inv[cls(i + 1, j, k)];
            }
            par |= ((j + k) & 1) << q;
        }
    }
    // off-diagonal sum at offset at (PER: of cell (i, j, k))
    __device__ __forceinline__ float offdiag(const float* x, int i, int j, int k) const {
        int w = -1, e = 1, s = -s1, n = s1, d = -s2, u = s2;
        if (PER) {
            if (L.per[0]) { if (i == 0) w = L.n[0] - 1; if (i == L.n[0] - 1) e = 1 - L.n[0]; }
            if (L.per[1]) { if (j == 0) s = (L.n[1] - 1) * s1; if (j == L.n[1] - 1) n = (1 - L.n[1]) * s1; }
            if (ND > 2 && L.per[2]) { if (k == 0) d = (L.n[2] - 1) * s2; if (k == L.n[2] - 1) u = (1 - L.n[2]) * s2; }
        }
        float acc = __fmaf_rn(c[0], x[w], 0.f);
        acc = __fmaf_rn(c[1], x[e], acc);
        acc = __fmaf_rn(c[2], x[s], acc);
        acc = __fmaf_rn(c[3], x[n], acc);
        if (ND > 2) {
            acc = __fmaf_rn(c[ND > 2 ? 4 : 0], x[d], acc);
            acc = __fmaf_rn(c[ND > 2 ? 5 : 0], x[u], acc);
        }
        return acc;
    }
    __device__ __forceinline__ void half(int color) const {
        float* x = sm + L.x;
        const float* b = sm + L.b;
#pragma unroll 1
        for (int q = 0; q < cnt; ++q) {
            const int e = ((par >> q) ^ color) & 1, at = o[q] + e;  // the pair's cell of this colour
            const float iv = inv[q][e];
            int t = 0, j = 0, k = 0;
            if (PER) place(q, t, j, k);
            if (iv != 0.f) x[at] = __fmul_rn(__fsub_rn(b[at], offdiag(x + at, 2 * t + e, j, k)), iv);
        }
        sync();
    }
    __device__ __forceinline__ float residual(int i, int j, int k, int at) const {
        const float* x = sm + L.x + at;
        return __fsub_rn(sm[L.b + at], __fmaf_rn(L.c0[cls(i, j, k)], *x, offdiag(x, i, j, k)));
    }

    // pre-smoothing from x = 0, the residual and its restriction
    __device__ __forceinline__ void down(const SmLevel& Lc, int sweeps, float* r) const {
        if (warp >= act) return;
        // (the first half sweep from zero: x = b / c0; the other colour's x is 0 already)
#pragma unroll 1
        for (int q = 0; q < cnt; ++q) {
            const int e = (par >> q) & 1, at = o[q] + e;
            const float iv = inv[q][e];
            if (iv != 0.f) sm[L.x + at] = __fmul_rn(sm[L.b + at], iv);
        }
        sync();
#pragma unroll 1
        for (int h = 1; h < 2 * sweeps; ++h) half(h & 1);
        float* bc = sm + Lc.b;
        const int nc0 = Lc.n[0], nc1 = Lc.n[1];
        if (!Lc.node) {
            // the average of the children that exist, or with all's weight (warps take 2^lf cells of 32 / 2^lf rows)
            const int lf = Lc.lf, groups = Lc.fgroups, rows = Lc.frows, total = groups * rows * (ND > 2 ? Lc.n[2] : 1);
            for (int g = warp; g < total; g += act) {
                const int rg = groups == 1 ? g : g / groups, K = ND > 2 ? small_div(rg, Lc.mfrows) : 0;
                const int I = ((g - rg * groups) << lf) + (lane & ((1 << lf) - 1)), J = ((rg - K * rows) << (5 - lf)) + (lane >> lf);
                if (I >= nc0 || J >= nc1) continue;
                float acc = 0.f;
                int n = 0;
#pragma unroll
                for (int q = 0; q < (1 << ND); ++q) {
                    const int i = 2 * I + (q & 1), j = 2 * J + ((q >> 1) & 1), k = ND > 2 ? 2 * K + (q >> 2) : 0;
                    if (i < L.n[0] && j < L.n[1] && (ND < 3 || k < L.n[2])) {
                        acc = __fadd_rn(acc, residual(i, j, k, i + j * s1 + (ND > 2 ? k * s2 : 0)));
                        ++n;
                    }
                }
                bc[I + J * Lc.s1 + (ND > 2 ? K * Lc.s2 : 0)] = __fmul_rn(acc, L.adjoint ? (ND > 2 ? 0.125f : 0.25f) : n == 8 ? 0.125f : n == 4 ? 0.25f : n == 2 ? 0.5f : 1.f);
            }
        } else {
#pragma unroll 1
            for (int q = 0; q < cnt; ++q) {
                int t, j, k;
                place(q, t, j, k);
#pragma unroll 1
                for (int e = 0; e < 2; ++e)
                    if (inv[q][e] != 0.f) r[o[q] + e] = residual(2 * t + e, j, k, o[q] + e);
            }
            sync();
            // full weighting: coarse node I <-> fine node 2 I
            const int total = nc0 * nc1 * (ND > 2 ? Lc.n[2] : 1);
            for (int g = (int) threadIdx.x; g < total; g += act * 32) {
                const int row = g / nc0, K = ND > 2 ? row / nc1 : 0, I = g - row * nc0, J = row - K * nc1;
                const int fi = 2 * (Lc.lo[0] + I) - L.lo[0], fj = 2 * (Lc.lo[1] + J) - L.lo[1], fk = ND > 2 ? 2 * (Lc.lo[2] + K) - L.lo[2] : 0;
                float acc = 0.f;
#pragma unroll
                for (int dz = ND > 2 ? -1 : 0; dz <= (ND > 2 ? 1 : 0); ++dz)
#pragma unroll
                    for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
                        for (int dx = -1; dx <= 1; ++dx) {
                            const float w = (dx == 0 ? 0.5f : 0.25f) * (dy == 0 ? 0.5f : 0.25f) * (ND > 2 ? (dz == 0 ? 0.5f : 0.25f) : 1.f);
                            const int i = fi + dx, j = fj + dy, k = fk + dz;
                            if ((unsigned) i < (unsigned) L.n[0] && (unsigned) j < (unsigned) L.n[1] && (ND < 3 || (unsigned) k < (unsigned) L.n[2]))
                                acc = __fmaf_rn(w, r[i + j * s1 + (ND > 2 ? k * s2 : 0)], acc);
                        }
                bc[I + J * Lc.s1 + (ND > 2 ? K * Lc.s2 : 0)] = acc;
            }
        }
        sync();
    }

    // place (times the stride) of coarse index I along d by the ghost rules; f: turned or zeroed with it
    __device__ __forceinline__ int ghost(const SmLevel& Lc, int d, int I, float& f) const {
        const int st = d == 0 ? 1 : d == 1 ? Lc.s1 : Lc.s2;
        if ((unsigned) I < (unsigned) Lc.n[d]) return I * st;
        const int rule = I < 0 ? Lc.glo[d] : Lc.ghi[d];
        if (rule == GH_WRAP) return (I < 0 ? I + Lc.n[d] : I - Lc.n[d]) * st;
        if (rule == GH_ZERO) f = Lc.node ? 0.f : -f;
        return (I < 0 ? 0 : Lc.n[d] - 1) * st;
    }
    // the two coarse places and factors along d for fine index i of a cell- or node-centred level
    __device__ __forceinline__ void two(const SmLevel& Lc, int d, int i, int (&at)[2], float (&sg)[2], float (&w)[2]) const {
        int I, J;
        if (!Lc.node) {
            I = i >> 1;
            J = (i & 1) ? I + 1 : I - 1;
            w[0] = 0.75f;
            w[1] = 0.25f;
        } else {
            const int g = L.lo[d] + i, odd = g & 1;
            I = ((g - odd) >> 1) - Lc.lo[d];
            J = I + odd;
            w[0] = odd ? 0.5f : 1.f;
            w[1] = odd ? 0.5f : 0.f;
        }
        sg[0] = sg[1] = 1.f;
        at[0] = ghost(Lc, d, I, sg[0]);
        at[1] = ghost(Lc, d, J, sg[1]);
    }

    // prolongation and post-smoothing
    __device__ __forceinline__ void up(const SmLevel& Lc, int sweeps) const {
        if (warp >= act) return;
        float* x = sm + L.x;
        const float* xc = sm + Lc.x;
#pragma unroll 1
        for (int q = 0; q < cnt; ++q) {
            int t, j, k;
            place(q, t, j, k);
            if (2 * t >= L.n[0] || j >= L.n[1]) continue;
            const int oq = 2 * t + j * s1 + (ND > 2 ? k * s2 : 0);
            int ay[2], az[2] = {0, 0};
            float sy[2], wy[2], sz[2] = {1.f, 1.f}, wz[2] = {1.f, 0.f};
            two(Lc, 1, j, ay, sy, wy);
            if (ND > 2) two(Lc, 2, k, az, sz, wz);
#pragma unroll 1
            for (int e = 0; e < 2; ++e) {
                if (2 * t + e >= L.n[0]) continue;
                int ax[2];
                float sx[2], wx[2];
                two(Lc, 0, 2 * t + e, ax, sx, wx);
                float acc = 0.f;
#pragma unroll
                for (int m = 0; m < (1 << ND); ++m) {
                    const int ex = m & 1, ey = (m >> 1) & 1, ez = m >> 2;
                    const float w = __fmul_rn(__fmul_rn(wx[ex], wy[ey]), ND > 2 ? wz[ez] : 1.f);
                    const float s = sx[ex] * sy[ey] * (ND > 2 ? sz[ez] : 1.f);
                    acc = __fmaf_rn(w, __fmul_rn(s, xc[ax[ex] + ay[ey] + (ND > 2 ? az[ez] : 0)]), acc);  // (s: 1, -1 or 0)
                }
                x[oq + e] = __fadd_rn(x[oq + e], acc);
            }
        }
        sync();
#pragma unroll 1
        for (int h = 0; h < 2 * sweeps; ++h) half((h + 1) & 1);
    }
};

template <int ND, bool PER>
__device__ void small_vcycle(int pre, int post, float* sm, const SmProblem& P) {
    const int tid = threadIdx.x, warp = tid >> 5, nl = P.levels;
    const int n0 = P.lv[0].n[0], n1 = P.lv[0].n[1], cells = n0 * n1 * (ND > 2 ? P.lv[0].n[2] : 1);
    auto place0 = [&](int c) {  // cell c of the first level, in its frame
        const int row = small_div(c, P.mn0), k = ND > 2 ? small_div(row, P.lv[0].mrow) : 0;
        return c - row * n0 + (row - k * n1) * P.lv[0].s1 + (ND > 2 ? k * P.lv[0].s2 : 0);
    };
    {
        float* b = sm + P.lv[0].b;
#pragma unroll 4
        for (int c = tid; c < cells; c += SM_THREADS) b[place0(c)] = P.b[c];
    }
    __syncthreads();
    float* r = sm + P.frames + 1 + P.lv[0].s1 + P.lv[0].s2;  // (node-centred problems)
#pragma unroll 1
    for (int l = 0; l + 1 < nl; ++l) Small<ND, PER>(P.lv[l], sm).down(P.lv[l + 1], pre, r);
    __syncthreads();
    // the dense coarsest solve, accumulated in float64: eight lanes share a row
    {
        const SmLevel& L = P.lv[nl - 1];
        const int N = L.n[0] * L.n[1] * L.n[2];
        auto place = [&](int c) {
            const int q = c / L.n[0], k = ND > 2 ? q / L.n[1] : 0;
            return (c - q * L.n[0]) + (q - k * L.n[1]) * L.s1 + (ND > 2 ? k * L.s2 : 0);
        };
        double* lin = (double*) (sm + P.lin);  // b in the rows' order, converted once per entry
        for (int c = tid; c < N; c += SM_THREADS) lin[c] = (double) sm[L.b + place(c)];
        __syncthreads();
#pragma unroll 1
        for (int base = 0; base < N; base += SM_THREADS / 8) {
            const int row = base + tid / 8;
            double acc = 0.;
            if (row < N) {
                const double* Ar = P.Ainv + (long long) row * N;
#pragma unroll 8
                for (int col = tid & 7; col < N; col += 8) acc = fma(Ar[col], lin[col], acc);
            }
            for (int w = 4; w > 0; w >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, w);
            if (row < N && (tid & 7) == 0) sm[L.x + place(row)] = (float) acc;
        }
        __syncthreads();
    }
#pragma unroll 1
    for (int l = nl - 2; l >= 0; --l) {
        const int act = min(P.lv[l].shares, SM_WARPS);
        if (l < nl - 2 && warp < act) small_sync(act, P.lv[l].barrier);  // (the levels below are finished)
        Small<ND, PER>(P.lv[l], sm).up(P.lv[l + 1], post);
    }
    __syncthreads();
    const float* x = sm + P.lv[0].x;
#pragma unroll 4
    for (int c = tid; c < cells; c += SM_THREADS) P.x[c] = x[place0(c)];
}

__global__ void __launch_bounds__(SM_THREADS, 1) mg_small(const LvlDev* __restrict__ Ls, const int* __restrict__ top, const SmProblem* __restrict__ probs,
                                                         const Scal* sc, int pre, int post) {
    extern __shared__ float small_sm[];
    __shared__ SmProblem P;
    {
        const int* src = (const int*) (probs + blockIdx.x);
        for (int q = threadIdx.x; q < (int) (sizeof(SmProblem) / 4); q += SM_THREADS) ((int*) &P)[q] = src[q];
    }
    __syncthreads();
    if (sc && !sc[P.problem].active) return;  // (the whole CTA)
    for (int q = threadIdx.x; q < P.frames; q += SM_THREADS) small_sm[q] = 0.f;
    if (P.restricts) {  // (the finer level's residual is where the chunked kernels leave it)
        const LvlDev& L = Ls[top[blockIdx.x]];
        for (int c = threadIdx.x; c < (int) L.N; c += SM_THREADS) {
            const int q = c / L.n[0], k = q / L.n[1];
            cell_restrict<float>(Ls, L, c - q * L.n[0], q - k * L.n[1], k);
        }
    }
    __syncthreads();
    if (P.ndim == 3) {
        if (P.per) small_vcycle<3, true>(pre, post, small_sm, P);
        else small_vcycle<3, false>(pre, post, small_sm, P);
    } else {
        if (P.per) small_vcycle<2, true>(pre, post, small_sm, P);
        else small_vcycle<2, false>(pre, post, small_sm, P);
    }
}

// The levels from `L` (and the next `levels` - 1) laid out for the kernel; false where they do not fit.
bool mg_small_problem(const SmSource* L, int levels, const double* Ainv, SmProblem* P, long long* floats) {
    if (levels < 2 || levels > MG_BOTTOM_LEVELS) return false;
    std::memset(P, 0, sizeof *P);
    P->levels = levels;
    P->ndim = L[0].ndim;
    P->Ainv = Ainv;
    long long frames = 0;
    for (int q = 0; q < levels; ++q) {
        const SmSource& S = L[q];
        SmLevel& D = P->lv[q];
        for (int d = 0; d < 3; ++d) {
            D.n[d] = d < S.ndim ? S.n[d] : 1;
            D.lo[d] = S.lo[d];
            D.per[d] = S.per[d];
            D.glo[d] = S.glo[d];
            D.ghi[d] = S.ghi[d];
            P->per |= d < S.ndim && S.per[d];
        }
        const bool three = S.ndim > 2;
        D.s1 = (D.n[0] + 3) & ~1;  // (even: see the banks)
        D.s2 = three ? D.s1 * (D.n[1] + 2) : 0;
        const long long frame = (long long) D.s1 * (D.n[1] + 2) * (three ? D.n[2] + 2 : 1);
        D.x = (int) frames + 1 + D.s1 + D.s2;
        D.b = D.x + (int) frame;
        frames += 2 * frame;
        if (frames > MG_SMALL_FLOATS) return false;
        D.barrier = 1 + q;
        D.node = S.node;
        D.adjoint = S.adjoint;
        P->node |= S.node;
        auto magic = [](unsigned d) { return 0xFFFFFFFFu / d + 1; };  // (d = 1: 0)
        const int hw = (D.n[0] + 1) / 2;
        D.lw = hw <= 4 ? 2 : hw <= 8 ? 3 : 4;
        D.half = (hw + (1 << D.lw) - 1) >> D.lw;
        D.pairs = (D.n[1] + (32 >> D.lw) - 1) / (32 >> D.lw);
        D.mhalf = magic(D.half);
        D.mrows = magic(D.pairs);
        D.lf = D.n[0] <= 4 ? 2 : D.n[0] <= 8 ? 3 : D.n[0] <= 16 ? 4 : 5;
        D.fgroups = (D.n[0] + (1 << D.lf) - 1) >> D.lf;
        D.frows = (D.n[1] + (32 >> D.lf) - 1) / (32 >> D.lf);
        D.mfrows = magic(D.frows);
        D.mrow = magic(D.n[1]);
        D.shares = D.half * D.pairs * D.n[2];
        if (q + 1 < levels) {
            if (D.shares > MG_SMALL_SHARES * SM_WARPS) return false;
            for (int k = 0; k < 6; ++k) D.c[k] = (float) (*S.tab)[(three ? 13 : 4) * NSLOT + 1 + k];
            for (int k = 0; k < (three ? 27 : 9); ++k) {
                D.c0[k] = (float) (*S.tab)[k * NSLOT];
                if (D.c0[k] == 0.f) return false;
                D.inv[k] = 1.0f / D.c0[k];
                if (D.inv[k] == 0.f) return false;  // (0 stands for no cell)
            }
        }
    }
    P->frames = (int) frames;
    P->lin = ((int) frames + (P->node ? P->lv[0].b - P->lv[0].x : 0) + 1) & ~1;
    P->mn0 = 0xFFFFFFFFu / P->lv[0].n[0] + 1;
    const SmLevel& C = P->lv[levels - 1];
    *floats = P->lin + 2LL * C.n[0] * C.n[1] * C.n[2];
    return *floats <= MG_SMALL_FLOATS;
}

int mg_launch_small(cudaStream_t s, const LvlDev* L, const int* top, const SmProblem* probs, int ntop, const Scal* sc, int pre, int post, long long floats) {
    if (ntop <= 0) return OPFLOW_OK;
    if (floats > MG_SMALL_FLOATS) return fail(OPFLOW_E_INVALID, "small levels of %lld values (limit %lld)", floats, MG_SMALL_FLOATS);
    OPG_CUDA(cudaFuncSetAttribute(mg_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) (MG_SMALL_FLOATS * sizeof(float))));
    mg_small<<<ntop, SM_THREADS, (size_t) floats * sizeof(float), s>>>(L, top, probs, sc, pre, post);
    OPG_LAUNCHED();
    return check_launch("mg_small");
}

}  // namespace opg
