// Scalar programs (tape.h): building and running.
//
// An interpreted operation costs a few tens of issue slots for its fetch, its dispatch and its operands in
// shared memory; a float64 operation holds the SM's float64 pipe for 16 cycles = 64 issue slots.  So what
// bounds a program is its float64 operations, and those are what the builder saves, changing no bit:
//  - equal operations on equal values are formed once (a difference operator's left and right neighbours,
//    the spacings and positions of an interpolation);
//  - values of one direction's mesh positions alone are tabulated, once per index instead of once per cell;
//  - a division is six operations given the divisor's reciprocal (div_rn: the IEEE quotient), two where the
//    divisor is a constant (DIVC), none for a power of two, as its multiplications are (the exponent moves);
//  - products with 1 and -1 are not formed.
// A thread takes a cell; the values live at one time stand in shared memory, a column per thread.
// Measured against the stack program over the expanded tree (a thread per cell, stack in local memory):
// variable-coefficient transport, 1000 x 702, 315 -> 137 us per step (168 -> 76 float64 operations per cell, the
// pipe 63 % busy); coefficients of the 3D flux-form equation at 192^3 8.5 -> 1.5 ms.  With the program in global
// memory instead of the kernel's parameters 163 us, with one cell per thread 168.
#include "tape.h"
#include "f64div.h"
#include "pointwise.h"
#include "stencil.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <functional>

namespace opg {

constexpr int TP_THREADS = 128;
constexpr int TP_SLOTS = 40;    // values live at once: 40 KB of shared memory per CTA, five CTAs per SM
constexpr int TP_CONSTS = 896;  // with the values below 48 KB
constexpr int TP_CODE_SMALL = 124, TP_CODE = 640;  // instructions of a launch: 4 KB and 20 KB of kernel parameters

// ======================================================================================== builder
static long long bits_of(double v) {
    long long b;
    std::memcpy(&b, &v, sizeof b);
    return b;
}

unsigned long long Tape::hash(const Node& n) {
    unsigned long long h = (unsigned long long) bits_of(n.v) ^ (unsigned long long) n.lin * 0x9E3779B97F4A7C15ull;
    h = (h ^ (h >> 32)) * 0xBF58476D1CE4E5B9ull + ((unsigned long long) n.op << 40 | (unsigned long long) n.slot << 48);
    h = (h ^ (unsigned) n.a ^ (unsigned long long) (unsigned) n.b << 20 ^ (unsigned long long) (unsigned) n.c << 40) * 0x94D049BB133111EBull;
    return h ^ (h >> 31);
}

int Tape::intern(const Node& n) {
    if (2 * nodes_.size() >= index_.size()) {  // (at least half of it free)
        index_.assign(std::max<size_t>(256, 2 * index_.size()), -1);
        for (size_t q = 0; q < nodes_.size(); ++q) {
            size_t at = hash(nodes_[q]) & (index_.size() - 1);
            while (index_[at] >= 0) at = (at + 1) & (index_.size() - 1);
            index_[at] = (int) q;
        }
    }
    size_t at = hash(n) & (index_.size() - 1);
    for (; index_[at] >= 0; at = (at + 1) & (index_.size() - 1)) {
        const Node& m = nodes_[index_[at]];
        if (m.op == n.op && m.slot == n.slot && m.a == n.a && m.b == n.b && m.c == n.c && m.lin == n.lin && bits_of(m.v) == bits_of(n.v)) return index_[at];
    }
    index_[at] = (int) nodes_.size();
    nodes_.push_back(n);
    per_cell_ += n.op != T_CONST && n.op != T_NEG && n.dep != 1 && n.dep != 2 && n.dep != 4;
    return index_[at];
}
bool Tape::too_long() const { return per_cell_ > TP_CODE; }

int Tape::cst(double v) { return intern(Node{T_CONST, 0, -1, -1, -1, 0, v, 0}); }
int Tape::load(int slot, const FieldView& f, const int* off) {
    return intern(Node{T_LOAD, slot, -1, -1, -1, off[0] + off[1] * (long long) f.sy + off[2] * (long long) f.sz, 0., 8 | (256 << slot)});
}
int Tape::pos(int op, int d, int o) { return intern(Node{op, d, -1, -1, -1, o, 0., 1 << d}); }

bool Tape::is_const(int id, double* v) const {
    if (nodes_[id].op != T_CONST) return false;
    *v = nodes_[id].v;
    return true;
}

int Tape::direction(int id) const {
    const int d = nodes_[id].dep;
    return d == 1 ? 0 : d == 2 ? 1 : d == 4 ? 2 : -1;
}

std::vector<char> Tape::formed_from(int id) const {
    std::vector<char> in(id + 1, 0);
    in[id] = 1;
    for (int q = id; q >= 0; --q)  // (operands come first)
        for (int o : {nodes_[q].a, nodes_[q].b, nodes_[q].c})
            if (o >= 0 && in[q]) in[o] = 1;
    return in;
}

int Tape::node(int op, int slot, int a, int b, int c) {
    Node n{op, slot, a, b, c, 0, 0., 0};
    for (int q : {a, b, c})
        if (q >= 0) n.dep |= nodes_[q].dep;
    return intern(n);
}

int Tape::neg(int a) {
    double v;
    if (is_const(a, &v)) return cst(-v);
    if (nodes_[a].op == T_NEG) return nodes_[a].a;
    return node(T_NEG, 0, a);
}

// the exponent k of a positive power of two in the range that T_SHL takes
static bool pow2_shift(double v, int* k) {
    int e;
    if (!(v > 0) || !std::isfinite(v) || std::frexp(v, &e) != 0.5 || e < -400 || e > 400) return false;
    *k = e - 1;
    return true;
}

int Tape::bin(int op, int a, int b) {
    double x = 0., y = 0.;
    const bool ca = is_const(a, &x), cb = is_const(b, &y);
    int k;
    if (op == T_ADD || op == T_SUB || op == T_MUL || op == T_DIV) {
        if (ca && cb) return cst(op == T_ADD ? x + y : op == T_SUB ? x - y : op == T_MUL ? x * y : x / y);
        if (op == T_DIV && cb && pow2_shift(y, &k)) return bin(T_MUL, a, cst(1.0 / y));
        if (op == T_MUL && ca) {
            std::swap(a, b);
            std::swap(x, y);
        }
        if (op == T_MUL && (ca || cb)) {  // (y: the constant, now b)
            if (y == 1.) return a;
            if (y == -1.) return neg(a);
            if (pow2_shift(y, &k)) {
                Node n{T_SHL, 0, a, -1, -1, k, 0., nodes_[a].dep};
                return intern(n);
            }
        }
        if (op == T_ADD && nodes_[b].op == T_NEG) return bin(T_SUB, a, nodes_[b].a);
        if (op == T_ADD && nodes_[a].op == T_NEG) return bin(T_SUB, b, nodes_[a].a);
        if (op == T_SUB && nodes_[b].op == T_NEG) return bin(T_ADD, a, nodes_[b].a);
        if ((op == T_ADD || op == T_MUL) && a > b) std::swap(a, b);
        if (op == T_DIV) {
            AxisParams P;
            int e;
            std::frexp(y, &e);
            if (cb && y > 0 && std::isfinite(y) && std::abs(e) < 100 && axis_divisor(&P, 0, y) && !P.pow2[0]) {
                Node n{T_DIVC, 0, a, -1, -1, 0, y, nodes_[a].dep};
                return intern(n);
            }
            return node(T_DIV, 0, a, b, cb ? cst(1.0 / y) : node(T_RCP, 0, b));
        }
    }
    return node(op, 0, a, b);
}

int Tape::const_at(const std::vector<double>& block) {
    std::vector<long long> key;
    for (double v : block) key.push_back(bits_of(v));
    auto it = const_index_.find(key);
    if (it != const_index_.end()) return it->second;
    const int at = (int) consts_.size();
    consts_.insert(consts_.end(), block.begin(), block.end());
    return const_index_[key] = at;
}

// operands first, depth first, so that values live shortly; a place is reused once its value was read last
bool Tape::emit(const std::vector<Out>& outs, const std::vector<int>& tab, Program* P) {
    std::vector<int> order, uses(nodes_.size(), 0), state(nodes_.size(), 0);
    std::function<void(int)> visit = [&](int id) {
        if (id < 0 || state[id] || nodes_[id].op == T_CONST) return;
        state[id] = 1;
        const Node& n = nodes_[id];
        if (!tab[id])
            for (int q : {n.a, n.b, n.c}) visit(q);
        order.push_back(id);
    };
    struct Step { int id; Out out; };
    std::vector<Step> steps;
    for (const Out& o : outs) {
        order.clear();
        visit(o.id);
        for (int id : order) steps.push_back({id, {}});
        if (o.op != T_CONST) steps.push_back({-1, o});
    }
    for (const Step& s : steps) {
        if (s.id < 0) { ++uses[s.out.id]; continue; }
        if (tab[s.id]) continue;
        for (int q : {nodes_[s.id].a, nodes_[s.id].b, nodes_[s.id].c})
            if (q >= 0) ++uses[q];
    }
    std::vector<int> place(nodes_.size(), -1), free_places;
    int slots = 0;
    const int row = TP_THREADS * 8;
    auto operand = [&](int id) -> int {
        if (id < 0) return 0;
        if (nodes_[id].op == T_CONST) return ~(8 * const_at({nodes_[id].v}));
        return place[id] * row;
    };
    auto done = [&](int id) {
        if (id >= 0 && nodes_[id].op != T_CONST && --uses[id] == 0) free_places.push_back(place[id]);
    };
    for (const Step& s : steps) {
        TInstr in{};
        if (s.id < 0) {
            in.op = s.out.op;
            in.slot = s.out.slot;
            in.a = operand(s.out.id);
            if (in.op == T_TABOUT) in.lin = tab_first_[s.out.id];
            P->code.push_back(in);
            done(s.out.id);
            continue;
        }
        const Node& n = nodes_[s.id];
        in.op = n.op;
        in.slot = n.slot;
        in.lin = n.lin;
        if (tab[s.id]) {
            in.op = T_TAB;
            in.lin = tab_first_[s.id];
            in.slot = direction(s.id);
        } else {
            in.a = operand(n.a);
            in.b = operand(n.b);
            in.c = operand(n.c);
            if (n.op == T_DIVC) {
                AxisParams A;
                axis_divisor(&A, 0, n.v);
                const long long bad = A.guard[0] ? ((long long) A.bad_hi[0] << 32 | (unsigned) A.bad_lo[0]) : -1;
                double bd;
                std::memcpy(&bd, &bad, 8);
                in.b = 8 * const_at({A.inv_h[0], A.cl[0], n.v, bd});
            }
            done(n.a);
            done(n.b);
            done(n.c);
        }
        if (free_places.empty()) place[s.id] = slots++;
        else {
            place[s.id] = free_places.back();
            free_places.pop_back();
        }
        in.dst = place[s.id] * row;
        P->code.push_back(in);
        if (uses[s.id] == 0) free_places.push_back(place[s.id]);
    }
    P->slots = std::max(slots, 1);
    return slots <= TP_SLOTS && (int) consts_.size() <= TP_CONSTS;
}

bool Tape::finish(const Box& box, bool hoist) {
    // the values that go to tables: of one direction, formed by float64 operations, and read by others
    std::vector<int> tab(nodes_.size(), 0), none(nodes_.size(), 0), root(nodes_.size(), 0);
    tab_first_.assign(nodes_.size(), -1);
    std::vector<Out> touts[3];
    if (hoist) {
        std::vector<int> need(nodes_.size(), 0);
        for (const Out& o : outs_) need[o.id] = 1, root[o.id] = 1;
        for (int id = (int) nodes_.size() - 1; id >= 0; --id) {
            if (!need[id]) continue;
            const Node& n = nodes_[id];
            if (direction(id) >= 0 && n.op != T_X && n.op != T_DX) { tab[id] = 1; continue; }
            for (int q : {n.a, n.b, n.c})
                if (q >= 0) need[q] = 1;
        }
        for (int id = 0; id < (int) nodes_.size(); ++id)
            if (tab[id]) {
                const int d = direction(id);
                tab_first_[id] = tab_entries_;
                tab_entries_ += box.hi[d] - box.lo[d];
                touts[d].push_back({T_TABOUT, d, id});
            }
    }
    for (int d = 0; d < 3; ++d)
        if (!touts[d].empty() && !emit(touts[d], none, &table_[d])) return false;
    return emit(outs_, tab, &main_) && main_.code.size() <= (size_t) TP_CODE &&
           table_[0].code.size() + table_[1].code.size() + table_[2].code.size() <= (size_t) TP_CODE;
}

// ======================================================================================== device
// (float64 operations of rarely taken branches, apart: predicated off they would hold the pipe all the same)
static __device__ __noinline__ double mul_apart(double a, double b) { return __dmul_rn(a, b); }
static __device__ __noinline__ double arith_apart(int arith, double o, double v) {
    switch (arith) {
        case OPFLOW_ASSIGN_ADD: return __dadd_rn(o, v);
        case OPFLOW_ASSIGN_SUB: return __dsub_rn(o, v);
        case OPFLOW_ASSIGN_MUL: return __dmul_rn(o, v);
        case OPFLOW_ASSIGN_DIV: return __ddiv_rn(o, v);
        default: return v;
    }
}

// gridDim.y programs (the tables of up to three directions in one launch, else one), as a kernel parameter:
// an instruction's fetch and dispatch are then uniform-datapath work
struct TapeHead {
    int first[4], slots[3];  // program y: code[first[y]] .. code[first[y + 1] - 1]
    Box box[3];
    const double* consts;
    int nconsts;
};
template <int CAP>
struct TapeConst : TapeHead {
    TInstr code[CAP];
};

// C cells per thread: an instruction's fetch and dispatch serve them all, and their chains overlap.
template <int C, int CAP>
__global__ void __launch_bounds__(TP_THREADS) tape_kernel(const __grid_constant__ TapeConst<CAP> T, const __grid_constant__ TapeArgs A) {
    extern __shared__ double tape_sm[];
    char* const sm = reinterpret_cast<char*>(tape_sm);
    for (int q = threadIdx.x; q < T.nconsts; q += TP_THREADS) tape_sm[q] = T.consts[q];
    __syncthreads();
    const int p0 = T.first[blockIdx.y], p1 = T.first[blockIdx.y + 1];
    const Box box = T.box[blockIdx.y];
    const int base = (T.nconsts + (int) threadIdx.x) * 8, per_cell = T.slots[blockIdx.y] * TP_THREADS * 8;
    // operand o of cell c
    auto get = [&](int o, int c) -> double { return *reinterpret_cast<const double*>(sm + (o < 0 ? ~o : o + base + c * per_cell)); };
    const long long total = box.count();
    for (long long t = blockIdx.x * (long long) (TP_THREADS * C) + threadIdx.x; t < total; t += (long long) gridDim.x * (TP_THREADS * C)) {
        int idx[C][3];
#pragma unroll
        for (int c = 0; c < C; ++c) {  // (a cell beyond the last is the last one again: the same values stored twice, T_OUT apart)
            const long long tc = t + c * TP_THREADS;
            box_index(tc < total ? tc : total - 1, box, idx[c][0], idx[c][1], idx[c][2]);
        }
#pragma unroll 1
        for (int p = p0; p < p1; ++p) {
            const TInstr& in = T.code[p];
            double r[C];
            auto at = [&](int c) { return in.slot == 0 ? idx[c][0] : in.slot == 1 ? idx[c][1] : idx[c][2]; };
#define EACH_CELL _Pragma("unroll") for (int c = 0; c < C; ++c)
            switch (in.op) {
                case T_LOAD: {
                    const FieldView& f = A.leaves[in.slot];
                    EACH_CELL r[c] = f.data[(idx[c][0] - f.off[0]) + (idx[c][1] - f.off[1]) * f.sy + (idx[c][2] - f.off[2]) * f.sz + in.lin];
                    break;
                }
                case T_X: EACH_CELL r[c] = A.x[in.slot][at(c) + (int) in.lin - A.es[in.slot]]; break;
                case T_DX: EACH_CELL r[c] = A.dx[in.slot][at(c) + (int) in.lin - A.es[in.slot]]; break;
                case T_TAB: EACH_CELL r[c] = A.tab[in.lin + at(c) - A.tab_box.lo[in.slot]]; break;
                case T_ADD: EACH_CELL r[c] = __dadd_rn(get(in.a, c), get(in.b, c)); break;
                case T_SUB: EACH_CELL r[c] = __dsub_rn(get(in.a, c), get(in.b, c)); break;
                case T_MUL: EACH_CELL r[c] = __dmul_rn(get(in.a, c), get(in.b, c)); break;
                case T_DIV: EACH_CELL r[c] = div_rn<true>(get(in.a, c), get(in.b, c), get(in.c, c)); break;
                case T_RCP: EACH_CELL r[c] = recip_fast(get(in.a, c)); break;
                case T_DIVC: {
                    const double* k = reinterpret_cast<const double*>(sm + in.b);
                    EACH_CELL {
                        const double x = get(in.a, c);
                        r[c] = __fma_rn(x, k[0], __dmul_rn(x, k[1]));
                        const long long xb = __double_as_longlong(x), m = xb & 0x7FFFFFFFFFFFFFFFll;
                        if (m == 0) r[c] = x;
                        else if ((unsigned) ((int) (m >> 52) - 150) > 1700u || (xb & 0xFFFFFFFFFFFFFll) == __double_as_longlong(k[3])) r[c] = div_apart(x, k[2]);
                    }
                    break;
                }
                case T_SHL: {
                    const int k = (int) in.lin;
                    EACH_CELL {
                        const double x = get(in.a, c);
                        const int hi = __double2hiint(x), lo = __double2loint(x), e = (hi >> 20) & 0x7FF;
                        r[c] = __hiloint2double(hi + k * (1 << 20), lo);
                        if (((hi & 0x7FFFFFFF) | lo) == 0) r[c] = x;
                        else if ((unsigned) (e - 1) >= 2046u || (unsigned) (e + k - 1) >= 2046u) r[c] = mul_apart(x, __hiloint2double((1023 + k) << 20, 0));
                    }
                    break;
                }
                case T_NEG: EACH_CELL r[c] = -get(in.a, c); break;
                case T_GT: EACH_CELL r[c] = get(in.a, c) > get(in.b, c) ? 1. : 0.; break;
                case T_GE: EACH_CELL r[c] = get(in.a, c) >= get(in.b, c) ? 1. : 0.; break;
                case T_LT: EACH_CELL r[c] = get(in.a, c) < get(in.b, c) ? 1. : 0.; break;
                case T_LE: EACH_CELL r[c] = get(in.a, c) <= get(in.b, c) ? 1. : 0.; break;
                case T_NE: EACH_CELL r[c] = get(in.a, c) != get(in.b, c) ? 1. : 0.; break;
                case T_AND: EACH_CELL r[c] = get(in.a, c) != 0. && get(in.b, c) != 0. ? 1. : 0.; break;
                case T_OR: EACH_CELL r[c] = get(in.a, c) != 0. || get(in.b, c) != 0. ? 1. : 0.; break;
                case T_NOT: EACH_CELL r[c] = get(in.a, c) == 0. ? 1. : 0.; break;
                case T_SEL: EACH_CELL r[c] = get(in.a, c) != 0. ? get(in.b, c) : get(in.c, c); break;
                case T_FIN: EACH_CELL r[c] = (__double2hiint(get(in.b, c)) & 0x7FF00000) == 0x7FF00000 ? __longlong_as_double(0x7FF8000000000000ll) : get(in.a, c); break;
                case T_F1: EACH_CELL r[c] = func1_eval(in.slot, get(in.a, c)); break;
                case T_F2: EACH_CELL r[c] = func2_eval(in.slot, get(in.a, c), get(in.b, c)); break;
                case T_LIM: EACH_CELL r[c] = flux_limiter(in.slot, get(in.a, c)); break;
                case T_OUT: {
                    const FieldView& o = A.out;
                    EACH_CELL {
                        const long long q = (idx[c][0] - o.off[0]) + (idx[c][1] - o.off[1]) * o.sy + (idx[c][2] - o.off[2]) * o.sz;
                        const double v = get(in.a, c);
                        // (`cur op value` in place is not to be applied twice)
                        if (c == 0 || t + c * TP_THREADS < total) o.data[q] = A.arith == OPFLOW_ASSIGN_EQ ? v : arith_apart(A.arith, A.cur.data[q], v);
                    }
                    continue;
                }
                case T_TABOUT: EACH_CELL A.tab[in.lin + at(c) - A.tab_box.lo[in.slot]] = get(in.a, c); continue;
                default: {  // T_COEF, T_RHS
                    const long long nx = A.rows.hi[0] - A.rows.lo[0], ny = A.rows.hi[1] - A.rows.lo[1];
                    EACH_CELL {
                        const long long q = (idx[c][0] - A.rows.lo[0]) + nx * ((idx[c][1] - A.rows.lo[1]) + ny * (idx[c][2] - A.rows.lo[2]));
                        const double v = get(in.a, c);
                        if (in.op == T_RHS) A.rhs[q] = v;
                        else A.coef[in.slot * A.rows.count() + q] = (__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFll) == 0 ? 0. : v;  // +0 for -0
                    }
                    continue;
                }
            }
            EACH_CELL *reinterpret_cast<double*>(sm + in.dst + base + c * per_cell) = r[c];
#undef EACH_CELL
        }
    }
}

// ======================================================================================== host
template <int CAP>
static void launch_cap(opflow_ctx ctx, const TapeHead& H, const std::vector<const std::vector<TInstr>*>& codes, const TapeArgs& A, int C, dim3 g, size_t sm) {
    TapeConst<CAP> T;
    static_cast<TapeHead&>(T) = H;
    int at = 0;
    for (const auto* code : codes) {
        std::copy(code->begin(), code->end(), T.code + at);
        at += (int) code->size();
    }
    if (C == 2) tape_kernel<2, CAP><<<g, TP_THREADS, sm, ctx->stream>>>(T, A);
    else tape_kernel<1, CAP><<<g, TP_THREADS, sm, ctx->stream>>>(T, A);
}

static int launch(opflow_ctx ctx, TapeHead& H, const std::vector<const std::vector<TInstr>*>& codes, const TapeArgs& A, int C, long long cells, int slots) {
    H.first[0] = 0;
    for (size_t q = 0; q < 3; ++q) H.first[q + 1] = H.first[q] + (q < codes.size() ? (int) codes[q]->size() : 0);
    const long long per = (long long) TP_THREADS * C;
    const dim3 g((unsigned) std::max(1LL, std::min((cells + per - 1) / per, (long long) ctx->num_sms * 64)), (unsigned) codes.size());
    const size_t sm = (size_t) H.nconsts * 8 + (size_t) slots * C * TP_THREADS * 8;
    if (H.first[3] <= TP_CODE_SMALL) launch_cap<TP_CODE_SMALL>(ctx, H, codes, A, C, g, sm);
    else launch_cap<TP_CODE>(ctx, H, codes, A, C, g, sm);
    OPG_LAUNCHED();
    return check_launch("tape_kernel");
}

int Tape::prepare(opflow_ctx ctx, const TapeArgs& A) {
    const size_t consts = (std::max<size_t>(consts_.size(), 1) * 8 + 255) / 256 * 256;
    blob_ = (char*) dev_alloc(ctx, consts + (size_t) tab_entries_ * 8 + 256);
    if (!blob_) return fail(OPFLOW_E_NOMEM, "expression program");
    off_tab_ = consts;
    if (!consts_.empty()) OPG_CUDA(cudaMemcpyAsync(blob_, consts_.data(), consts_.size() * 8, cudaMemcpyHostToDevice, ctx->stream));
    TapeHead H{};
    H.consts = (const double*) blob_;
    H.nconsts = (int) consts_.size();
    std::vector<const std::vector<TInstr>*> codes;
    int slots = 0;
    long long longest = 0;
    for (int d = 0; d < 3; ++d) {
        if (table_[d].code.empty()) continue;
        Box& box = H.box[codes.size()];
        box = A.tab_box;
        for (int e = 0; e < 3; ++e)
            if (e != d) box.hi[e] = box.lo[e] + 1;
        longest = std::max(longest, box.count());
        slots = std::max(slots, table_[d].slots);
        H.slots[codes.size()] = table_[d].slots;
        codes.push_back(&table_[d].code);
    }
    if (codes.empty()) return OPFLOW_OK;
    TapeArgs B = A;
    B.tab = (double*) (blob_ + off_tab_);
    return launch(ctx, H, codes, B, 1, longest, slots);
}

int Tape::run(opflow_ctx ctx, const TapeArgs& A) const {
    if (A.box.empty()) return OPFLOW_OK;
    TapeArgs B = A;
    B.tab = (double*) (blob_ + off_tab_);
    TapeHead H{};
    H.consts = (const double*) blob_;
    H.nconsts = (int) consts_.size();
    H.box[0] = A.box;
    H.slots[0] = main_.slots;
    // two cells per thread where two columns of values fit and the cells still fill the chip
    const int C = main_.slots <= TP_SLOTS / 2 && A.box.count() >= (long long) ctx->num_sms * TP_THREADS * 8 ? 2 : 1;
    return launch(ctx, H, {&main_.code}, B, C, A.box.count(), main_.slots);
}

void Tape::release(opflow_ctx ctx) {
    if (blob_) dev_free(ctx, blob_);
    blob_ = nullptr;
}

}  // namespace opg
