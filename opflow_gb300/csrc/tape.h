// Scalar programs over the cells of a box: an expression's or an equation's values as a list of operations
// on numbered values, each value formed once per cell (or once per index along one direction, where it
// depends on the mesh position along that direction alone).
#pragma once
#include "internal.h"

#include <array>
#include <map>
#include <vector>

namespace opg {

enum TOp : int {
    T_CONST = 0, T_LOAD, T_X, T_DX,
    T_ADD, T_SUB, T_MUL, T_DIV,  // (T_DIV: a, b and b's reciprocal)
    T_DIVC,                      // by a constant whose quotients two operations give (axis_divisor)
    T_SHL,                       // by a power of two
    T_RCP, T_NEG,
    T_GT, T_GE, T_LT, T_LE, T_NE, T_AND, T_OR, T_NOT, T_SEL,  // (T_SEL: a ? b : c)
    T_F1, T_F2, T_LIM,
    T_FIN,                       // a where b is finite, else NaN
    T_TAB,                       // a tabulated value of one direction
    T_OUT, T_COEF, T_RHS, T_TABOUT
};

struct TInstr {
    int op, slot;  // slot: leaf, direction, function or coefficient
    int dst;       // result: byte offset of its lane-0 place
    int a, b, c;   // operands: the same, or ~(byte offset) of a constant
    long long lin; // T_LOAD: offset from the cell; T_X, T_DX: along the direction; T_TAB(OUT): first entry; T_SHL: shift
};

struct TapeArgs {
    FieldView leaves[8];
    const double* x[3];
    const double* dx[3];
    int es[3];
    Box box;                // the cells run
    Box tab_box;            // the cells the tables cover
    double* tab;
    FieldView out, cur;     // T_OUT: out = value, or cur op value
    int arith;
    Box rows;               // T_COEF, T_RHS: the box whose cells number the entries
    double* coef;
    double* rhs;
};

// Builder: values are numbered as they are formed; equal operations on equal values are one value.  All the
// simplifications made here give the same bits as the operations they replace.
class Tape {
public:
    int cst(double v);
    int load(int slot, const FieldView& f, const int* off);
    int pos(int op, int d, int o);  // T_X, T_DX
    int bin(int op, int a, int b);  // T_ADD .. T_DIV, comparisons, T_AND, T_OR
    int neg(int a);
    int node(int op, int slot, int a, int b = -1, int c = -1);
    bool is_const(int id, double* v) const;
    int direction(int id) const;  // the direction whose mesh positions alone a value depends on, -1: none or several
    void out(int op, int slot, int id) { outs_.push_back({op, slot, id}); }
    void form(int id) { outs_.push_back({T_CONST, 0, id}); }  // here in the program, read by a later one
    std::vector<char> formed_from(int id) const;              // per value up to id: whether id is it or is formed from it
    unsigned fields(int id) const { return (unsigned) nodes_[id].dep >> 8; }  // the leaf slots that id is formed from, a bit each
    // Whether the values formed so far, each of them read by the program's result, are already more than the kernel
    // takes (constants, negations and values of one direction left out: they may go elsewhere); finish() is then false.
    bool too_long() const;
    // Lays the program out; `hoist`: values of one direction go to tables.  false: too long, or too many values
    // live at once, for the kernel.
    bool finish(const Box& box, bool hoist);
    // Allocates (dev_alloc) and fills the device side and the tables; run() launches over A.box.  The
    // arguments' leaves, mesh and tab_box have to be those of the launches.
    int prepare(opflow_ctx ctx, const TapeArgs& A);
    int run(opflow_ctx ctx, const TapeArgs& A) const;
    void release(opflow_ctx ctx);

private:
    struct Node { int op, slot, a, b, c; long long lin; double v; int dep; };  // dep: bit d: X or DX along d; bit 3: a field; bit 8 + s: leaf s
    struct Out { int op, slot, id; };
    struct Program { std::vector<TInstr> code; int slots = 0; };
    static unsigned long long hash(const Node& n);
    int intern(const Node& n);
    bool emit(const std::vector<Out>& outs, const std::vector<int>& tab, Program* P);
    int const_at(const std::vector<double>& block);
    std::vector<Node> nodes_;
    std::vector<int> index_;  // the values by their hash (open addressing, -1: free)
    std::vector<Out> outs_;
    std::vector<double> consts_;
    std::map<std::vector<long long>, int> const_index_;
    Program main_, table_[3];
    std::vector<long long> tab_first_;  // per value: first table entry, -1 none
    long long tab_entries_ = 0;
    int per_cell_ = 0;                  // values that only the cells' own program can form
    char* blob_ = nullptr;
    size_t off_tab_ = 0;
};

}  // namespace opg
