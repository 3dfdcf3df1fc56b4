// fn_jit.cpp -- code generation, NVRTC compilation and the module registry of
// the run-time specialised kernels (see fn_jit.h).
#include "fn_jit.h"

#include <nvrtc.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <deque>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <mutex>
#include <sstream>
#include <thread>
#include <unordered_map>
#include <unordered_set>

#include <sys/stat.h>
#include <unistd.h>

#include "FastNoise/FastNoise_C.h"
#include "fn_kernels.cuh"
#include "fn_runtime.h"

namespace fn {

// The device headers (fn_types.h, fn_device.cuh, fn_eval.cuh) as one source
// string; the file defining it is generated at build time (build.py).
const char* embedded_device_source();

namespace {

std::string lit(float f)
{
    char b[64];
    if (std::isfinite(f)) {
        std::snprintf(b, sizeof b, "%af", (double)f);         // exact hexadecimal literal
    } else {
        uint32_t u;
        std::memcpy(&u, &f, 4);
        std::snprintf(b, sizeof b, "__int_as_float(0x%08xu)", u);
    }
    return b;
}

std::string r(int i) { return "r" + std::to_string(i); }

constexpr int kColMaxRegs = 200;       // registers of column state a kernel may hold
constexpr int kColMaxTable = 370;       // float4 of shared table per warp (8 warps within 48 KB of static shared memory)

const char* noise_fn(int kind)
{
    switch (kind) {
    case FN_NOISE_SIMPLEX: return "simplex";
    case FN_NOISE_SUPERSIMPLEX: return "supersimplex";
    case FN_NOISE_PERLIN: return "perlin";
    default: return "value";
    }
}

// Column evaluation of a program over a uniform grid (fn_column.cuh): the noise
// instructions whose position is separable -- every component but the last depends on the
// grid's fixed axes only, the last on the column's axis only, all through constant scales
// and offsets -- keep their lattice state between the steps of a column.
struct ColState {
    int pc = 0;                        // instruction
    std::string type;                  // state struct of fn_column.cuh
    std::vector<std::string> pos;      // fixed components as expressions of the root position
    std::string along;                 // the last component, as an expression of the column's coordinate
    std::string jitter;                // cellular states: the jitter
    ColumnRate rate;                   // how often it is rebuilt, and at what cost
    int table = 0, table_size = 0;     // its part of the warp's shared table, in float4
};
struct ColPlan {
    std::vector<ColState> states;
    int regs = 0;                      // registers the states hold
    int table = 0;                     // float4 of shared table per warp
    float step = 0.0f, point = 0.0f;   // issue slots of a step, and of a point of the point kernel

    const ColState* at(int pc) const
    {
        for (auto& st : states) if (st.pc == pc) return &st;
        return nullptr;
    }
};

ColPlan column_plan(const CompiledProgram& prog)
{
    ColPlan plan;
    const FnProgramHeader* h = reinterpret_cast<const FnProgramHeader*>(prog.blob.data());
    const FnInstr* ins = fn_program_instrs(h);
    const float* P = fn_program_params(h);
    // what is known of a register: a constant, a function of the fixed axes (with its
    // expression), of the column's axis (with the product of its scales), or neither
    struct Reg {
        enum { kOther, kConst, kFixed, kColumn } kind = kOther;
        std::string expr;
        float scale = 0.0f;            // product of its scales (a constant's value)
        int axis = 0;                  // grid axis it depends on
    };
    std::vector<Reg> R((size_t)std::max<int>(h->n_regs, h->dim));
    const char* root[4] = {"x", "y", "z", "w"};
    for (int k = 0; k < h->dim; ++k) {
        R[(size_t)k].kind = k == h->dim - 1 ? Reg::kColumn : Reg::kFixed;
        R[(size_t)k].expr = root[k];
        R[(size_t)k].scale = 1.0f;
        R[(size_t)k].axis = k;
    }
    // Issue slots, fitted to the times of 2200 batches of random trees and grids (which they give
    // within about 9 %): of a point of the point kernel, of a step of each state, and of the rebuild
    // that entering a cell costs (a lattice plane, or a neighbourhood).  They choose the kernel.
    double step = 0, point = prog.dim == 2 ? 35 : prog.dim == 3 ? 65 : 80;
    auto generic_cost = [&](const FnInstr& I) -> double {
        const int d = I.dim - 2;
        static const double simplex[3] = {110, 200, 330}, super[3] = {175, 390, 900}, perlin[3] = {105, 180, 395}, value[3] = {55, 95, 185},
                            warp[3] = {85, 210, 500}, cells[3] = {480, 1500, 4000};
        switch (I.op) {
        case FN_OP_NOISE: return (I.aux == FN_NOISE_SIMPLEX ? simplex : I.aux == FN_NOISE_SUPERSIMPLEX ? super : I.aux == FN_NOISE_PERLIN ? perlin : value)[d];
        case FN_OP_WARP_GRAD: return warp[d];
        case FN_OP_WARP_SIMPLEX: return 2 * warp[d];
        case FN_OP_CELL_VALUE: case FN_OP_CELL_DIST: case FN_OP_CELL_LOOKUP: return cells[d];
        default: return 2.5;
        }
    };
    // a state for the instruction, if its position is separable and the kernel has room
    auto add_state = [&](int pc, const std::string& type, float freq, int regs, int table, bool cellular, double enter_cost,
                         double step_cost) -> ColState* {
        const FnInstr& I = ins[pc];
        bool ok = R[(size_t)(I.a + I.dim - 1)].kind == Reg::kColumn && plan.regs + regs <= kColMaxRegs &&
                  plan.states.size() < kMaxColumnStates && plan.table + table <= kColMaxTable;
        for (int k = 0; k < I.dim - 1; ++k)
            ok = ok && (R[(size_t)(I.a + k)].kind == Reg::kFixed || R[(size_t)(I.a + k)].kind == Reg::kConst);
        if (!ok) return nullptr;
        ColState st;
        st.pc = pc;
        st.type = type;
        st.rate.cellular = cellular;
        for (int k = 0; k < I.dim; ++k) {
            const Reg& r = R[(size_t)(I.a + k)];
            if (k < I.dim - 1) st.pos.push_back(r.expr + " * " + lit(freq));
            else st.along = r.expr + " * " + lit(freq);
            if (r.kind != Reg::kConst) st.rate.scale[r.axis] = std::max(st.rate.scale[r.axis], std::fabs(r.scale * freq));
        }
        st.table = plan.table;
        st.table_size = table;
        plan.table += table;
        plan.regs += regs;
        st.rate.enter = (float)enter_cost;
        st.rate.step = (float)step_cost;
        st.rate.point = (float)generic_cost(I);
        step += step_cost;
        plan.states.push_back(st);
        return &plan.states.back();
    };
    for (int pc = 0; pc < h->n_instr; ++pc) {
        const FnInstr& I = ins[pc];
        const int D = I.dim;
        const size_t had = plan.states.size();
        auto scaled = [&](const Reg& a, float f) {
            Reg r = a;
            if (r.kind == Reg::kConst) r.kind = Reg::kFixed;
            if (!r.expr.empty()) r.expr = "(" + r.expr + " * " + lit(f) + ")";
            r.scale *= f;
            return r;
        };
        auto set_other = [&](int reg, int n) { for (int k = 0; k < n; ++k) if (reg + k < (int)R.size()) R[(size_t)(reg + k)] = Reg(); };
        switch (I.op) {
        case FN_OP_CONST:
            R[I.dst] = Reg();
            R[I.dst].kind = Reg::kConst;
            R[I.dst].expr = lit(P[I.prm]);
            R[I.dst].scale = P[I.prm];
            break;
        case FN_OP_MOV: R[I.dst] = R[I.a]; break;
        case FN_OP_SCALE_POS: case FN_OP_SCALE_POS_V: {
            std::vector<Reg> t;
            for (int k = 0; k < D; ++k) t.push_back(scaled(R[(size_t)(I.a + k)], P[I.prm + (I.op == FN_OP_SCALE_POS_V ? k : 0)]));
            for (int k = 0; k < D; ++k) R[(size_t)(I.dst + k)] = t[(size_t)k];
            break;
        }
        case FN_OP_OFFSET_POS: {
            const int off[4] = {I.b, I.c, I.d, I.e};
            std::vector<Reg> t;
            for (int k = 0; k < D; ++k) {
                Reg r = R[(size_t)(I.a + k)];
                const Reg& o = R[(size_t)off[k]];
                if (r.kind == Reg::kConst) r.kind = Reg::kFixed;
                if (o.kind != Reg::kConst || r.kind == Reg::kOther) r = Reg();
                else r.expr = "(" + r.expr + " + " + o.expr + ")";
                t.push_back(r);
            }
            for (int k = 0; k < D; ++k) R[(size_t)(I.dst + k)] = t[(size_t)k];
            break;
        }
        case FN_OP_NOISE:
            if (I.aux == FN_NOISE_PERLIN)
                add_state(pc, "PerlinCol<" + std::to_string(D) + ">", P[I.prm], D == 2 ? 18 : D == 3 ? 20 : 38, 32, false,
                          D == 2 ? 127 : D == 3 ? 240 : 374, D == 2 ? 30 : D == 3 ? 32 : 90);
            else if (I.aux == FN_NOISE_VALUE)
                add_state(pc, "ValueCol<" + std::to_string(D) + ">", P[I.prm], 4, 32, false, D == 2 ? 60 : D == 3 ? 90 : 138, 5);
            R[I.dst] = Reg();
            break;
        case FN_OP_CELL_VALUE: case FN_OP_CELL_DIST: case FN_OP_CELL_LOOKUP: {
            // constant jitter, no size jitter, distances that are sums of squares (the 2D value
            // walk takes the root of Euclidean ones), the closest cell or two.  A jitter whose
            // square could overflow is left to the point function, which keeps its initial result
            // (hash or cell point 0) where every distance is infinite.
            const int df = I.aux & 15, slots = I.op == FN_OP_CELL_DIST ? std::max((I.aux >> 4) & 3, (I.aux >> 8) & 3) + 1 : ((I.aux >> 4) & 3) + 1;
            const Reg jit = R[I.b];
            const bool sums = df == 1 || (df == 0 && !(I.op == FN_OP_CELL_VALUE && D == 2));
            if (D < 4 && sums && jit.kind == Reg::kConst && std::fabs(jit.scale) <= 1e9f && I.c == FN_REG_NONE && I.d == FN_REG_NONE &&
                (I.op == FN_OP_CELL_LOOKUP || slots <= (I.op == FN_OP_CELL_DIST ? 2 : 1))) {
                const std::string kind = I.op == FN_OP_CELL_VALUE ? "kColValue" : I.op == FN_OP_CELL_DIST ? "kColDistance" : "kColLookup";
                // CellCol's part of the table (kTable there)
                const int cells = D == 3 ? 27 : 9, along = (D == 3 ? 12 : 4) * (I.op == FN_OP_CELL_LOOKUP ? 1 : 2);
                const int cell_table = 32 + 4 * cells + 3 * along + (I.op == FN_OP_CELL_VALUE ? cells : 0);
                ColState* st = add_state(pc, "CellCol<" + std::to_string(D) + ", fnd::" + kind + ", " + std::to_string(I.op == FN_OP_CELL_DIST ? slots : 1) + ">",
                                         P[I.prm], cells + 4, cell_table, true, D == 3 ? 640 : 120,
                                         I.op == FN_OP_CELL_DIST ? (D == 3 ? 203 : 113) : D == 3 ? 237 : 96);
                if (st) st->jitter = "fnd::CellConst<" + std::to_string(D) + ">::jitter * " + lit(jit.scale);
            }
            if (I.op == FN_OP_CELL_LOOKUP) set_other(I.dst, D);
            else R[I.dst] = Reg();
            break;
        }
        // in-place operands and multi-register results
        case FN_OP_SUB_POS: set_other(I.dst, D); break;
        case FN_OP_ROTATE2: set_other(I.dst, 2); break;
        case FN_OP_ROTATE3: set_other(I.dst, 3); break;
        case FN_OP_ROTPLANE: set_other(I.dst, std::max(3, D)); break;
        case FN_OP_WARP_GRAD: case FN_OP_WARP_SIMPLEX:
            if (I.op == FN_OP_WARP_GRAD && D < 4) {
                ColState* st = add_state(pc, "WarpCol<" + std::to_string(D) + ">", P[I.prm], D == 2 ? 4 : 6, 32 + (4 << D), true,
                                         D == 2 ? 60 : 170, D == 2 ? 40 : 110);
                if (st) st->jitter = "0.0f";
            }
            set_other(I.dst, D);
            if (I.c != FN_REG_NONE) set_other(I.c, 1);
            break;
        case FN_OP_FRACT_INIT: case FN_OP_FRACT_AMP: case FN_OP_FRACT_ACC: case FN_OP_DWF_AMP:
            set_other(I.dst, 1);
            if (I.a != FN_REG_NONE) set_other(I.a, 1);
            if (I.b != FN_REG_NONE) set_other(I.b, 1);
            break;
        default: set_other(I.dst, 1); break;
        }
        // the fewer warps of a column kernel hide less of the latency of 4D super-simplex' one copy
        const bool far = I.op == FN_OP_NOISE && I.aux == FN_NOISE_SUPERSIMPLEX && D == 4;
        if (plan.states.size() == had) step += (far ? 2.2 : 1.0) * generic_cost(I);
        point += generic_cost(I);
    }
    plan.step = (float)step;
    plan.point = (float)point;
    return plan;
}

// Statements that fill the shared gradient tables (fn_device.cuh) a kernel of `prog` reads: of
// the dimensionalities of its gradient noises, per-cell sub-programs included, but for those
// that are column states.
void gradient_dims(const CompiledProgram& prog, const ColPlan* col, bool* used)
{
    const FnProgramHeader* h = reinterpret_cast<const FnProgramHeader*>(prog.blob.data());
    const FnInstr* ins = fn_program_instrs(h);
    for (int pc = 0; pc < h->n_instr; ++pc)
        if (ins[pc].op == FN_OP_NOISE && ins[pc].aux != FN_NOISE_VALUE && !(col && col->at(pc))) used[ins[pc].dim] = true;
    for (auto& sub : prog.subs) gradient_dims(sub, nullptr, used);
}
std::string gradient_setup(const CompiledProgram& prog, const ColPlan* col = nullptr)
{
    bool used[5] = {};
    gradient_dims(prog, col, used);
    return std::string(used[3] ? "    fnd::gradient_init<3>();\n" : "") + (used[4] ? "    fnd::gradient_init<4>();\n" : "");
}

// One program -> `__device__ float <name>(int seed, float x, float y, float z, float w)`;
// with a column plan the function also takes the column's state, `struct <name>_state`.
// Its per-cell sub-programs (node-driven Minkowski P) come first, each as a
// function `<name>_s<j>` plus a functor `<name>_s<j>_mk` the cellular walk calls
// with the cell's offset vector.
void emit_eval(const CompiledProgram& prog, const std::string& name, std::ostringstream& o, const ColPlan* col = nullptr)
{
    const std::string sub_prefix = name + "_s";
    for (size_t j = 0; j < prog.subs.size(); ++j) {
        const std::string sub = sub_prefix + std::to_string(j);
        emit_eval(prog.subs[j], sub, o);
        const int sd = prog.subs[j].dim;
        o << "struct " << sub << "_mk {\n    int seed;\n    static constexpr bool kNode = true;\n"
          << "    __device__ __forceinline__ float operator()(const float* v) const { return " << sub << "(seed, v[0], v[1], "
          << (sd > 2 ? "v[2]" : "0.0f") << ", " << (sd > 3 ? "v[3]" : "0.0f") << "); }\n};\n\n";
    }
    const FnProgramHeader* h = reinterpret_cast<const FnProgramHeader*>(prog.blob.data());
    const FnInstr* ins = fn_program_instrs(h);
    const float* P = fn_program_params(h);
    const int nregs = h->n_regs;
    auto mk = [&](const FnInstr& I) {   // trailing functor argument of a cellular call
        return I.d == FN_REG_NONE ? std::string() : ", " + name + "_s" + std::to_string(I.d) + "_mk{seed}";
    };
    const char* root[4] = {"x", "y", "z", "w"};
    if (col) {
        o << "struct " << name << "_state {\n";
        for (auto& st : col->states) {
            o << "    fnd::" << st.type << " s" << st.pc << ";\n"
              << "    static __device__ __forceinline__ void pos" << st.pc << "(float x, float y, float z, float* q)\n    {\n"
              << "        x = fnd::opaque(x); y = fnd::opaque(y); z = fnd::opaque(z);\n";
            for (size_t k = 0; k < st.pos.size(); ++k) o << "        q[" << k << "] = " << st.pos[k] << ";\n";
            o << "    }\n";
        }
        const char* zc = root[h->dim - 1];
        o << "    __device__ __forceinline__ void init(float x, float y, float z)\n    {\n";
        for (auto& st : col->states)
            o << "        s" << st.pc << ".init([&](float* q) { pos" << st.pc << "(x, y, z, q); });\n";
        o << "    }\n    __device__ __forceinline__ unsigned prepare(float4* tab, unsigned lane, float " << zc << ")\n    {\n        return 0u";
        for (auto& st : col->states) o << " | s" << st.pc << ".prepare(tab + " << st.table << ", lane, " << st.along << ")";
        o << ";\n    }\n    __device__ __forceinline__ void enter(int seed, float4* tab, unsigned j, float x, float y, float z)\n    {\n";
        for (auto& st : col->states)
            o << "        s" << st.pc << ".enter(fnd::iadd(seed, " << ins[st.pc].seed << "), "
              << (st.rate.cellular ? "tab + " + std::to_string(st.table) + ", j, " + st.jitter : "tab[" + std::to_string(st.table) + " + j].w")
              << ", [&](float* q) { pos" << st.pc << "(x, y, z, q); });\n";
        o << "    }\n};\n";
    }
    o << "__device__ __forceinline__ float " << name << "(int seed, float x, float y, float z, float w"
      << (col ? ", const " + name + "_state& S, const float4* tab, unsigned j" : std::string()) << ")\n{\n";
    o << "    (void)x; (void)y; (void)z; (void)w;\n";
    for (int i = 0; i < nregs; ++i) o << "    float " << r(i) << " = " << (i < h->dim ? root[i] : "0.0f") << ";\n";
    // What is known of a register's value (beyond NaN): a constant, a noise output of bounded
    // size, the strength a gradient warp returned.  A weighted strength of constant 0 makes the
    // amplitude factor of an octave lerp(1, t, 0) = fma(0, t - 1, 1), which is 1 for every finite
    // t; a NaN t comes from a NaN noise (already in the sum) or NaN positions, so the result is
    // NaN with or without it.  The factor (and the warp's square root) is then left out:
    // FBm(Simplex) octaves lose 5 of ~150 instructions, a warp octave ~20 of ~190.
    enum Known { kUnknown, kConst, kBounded, kWarpStrength };
    struct { Known what = kUnknown; float value = 0.0f; } known[FN_MAX_REGS + 4];
    auto is_zero = [&](int reg) { return known[reg].what == kConst && known[reg].value == 0.0f; };
    for (int pc = 0; pc < h->n_instr; ++pc) {
        const FnInstr& I = ins[pc];
        const int D = I.dim;
        const std::string sd = "fnd::iadd(seed, " + std::to_string(I.seed) + ")";
        auto p = [&](int j) { return lit(P[I.prm + j]); };
        auto pos = [&](int base) {
            std::string s = "{";
            for (int j = 0; j < D; ++j) s += (j ? ", " : "") + r(base + j);
            return s + "}";
        };
        auto cellp = [&](int mk_index) {
            std::ostringstream c;
            c << "fnd::CellParams cp; cp.freq = " << p(0) << "; cp.jitter = fnd::CellConst<" << D << ">::jitter * " << r(I.b)
              << "; cp.sizeActive = " << (I.c != FN_REG_NONE ? "true" : "false") << "; cp.sizeJitter = "
              << (I.c != FN_REG_NONE ? r(I.c) + " * fnd::CellConst<" + std::to_string(D) + ">::size" : std::string("0.0f"))
              << "; cp.distFunc = " << (I.aux & 15) << "; cp.minkowski = " << p(mk_index) << ";";
            return c.str();
        };
        const ColState* cell = col ? col->at(pc) : nullptr;
        const std::string cell_state = "S.s" + std::to_string(pc), cell_tab = cell ? "tab + " + std::to_string(cell->table) + ", j" : std::string();
        auto fast = [&](const char* call) { return cell ? cell_state + ".fast ? " + cell_state + "." + call + cell_tab + ") : " : std::string(); };
        o << "    { // op " << (int)I.op << "\n";
        switch (I.op) {
        case FN_OP_CONST: o << "        " << r(I.dst) << " = " << p(0) << ";\n"; break;
        case FN_OP_MOV: o << "        " << r(I.dst) << " = " << r(I.a) << ";\n"; break;
        case FN_OP_SCALE_POS:
            for (int j = 0; j < D; ++j) o << "        const float t" << j << " = " << r(I.a + j) << " * " << p(0) << ";\n";
            for (int j = 0; j < D; ++j) o << "        " << r(I.dst + j) << " = t" << j << ";\n";
            break;
        case FN_OP_SCALE_POS_V:
            for (int j = 0; j < D; ++j) o << "        const float t" << j << " = " << r(I.a + j) << " * " << p(j) << ";\n";
            for (int j = 0; j < D; ++j) o << "        " << r(I.dst + j) << " = t" << j << ";\n";
            break;
        case FN_OP_OFFSET_POS: case FN_OP_SUB_POS: {
            const int off[4] = {I.b, I.c, I.d, I.e};
            const char* opch = I.op == FN_OP_OFFSET_POS ? " + " : " - ";
            for (int j = 0; j < D; ++j) o << "        const float t" << j << " = " << r(I.a + j) << opch << r(off[j]) << ";\n";
            for (int j = 0; j < D; ++j) o << "        " << r(I.dst + j) << " = t" << j << ";\n";
            break;
        }
        case FN_OP_ROTATE2:
            o << "        const float px = " << r(I.a) << ", py = " << r(I.a + 1) << ";\n";
            o << "        " << r(I.dst) << " = fmaf(-py, " << p(1) << ", px * " << p(0) << ");\n";
            o << "        " << r(I.dst + 1) << " = fmaf(px, " << p(1) << ", py * " << p(0) << ");\n";
            break;
        case FN_OP_ROTATE3:
            o << "        const float px = " << r(I.a) << ", py = " << r(I.a + 1) << ", pz = " << (D >= 3 ? r(I.a + 2) : "0.0f") << ";\n";
            for (int j = 0; j < 3; ++j)
                o << "        const float n" << j << " = fmaf(px, " << p(3 * j) << ", fmaf(py, " << p(3 * j + 1) << ", pz * " << p(3 * j + 2) << "));\n";
            for (int j = 0; j < 3; ++j) o << "        " << r(I.dst + j) << " = n" << j << ";\n";
            break;
        case FN_OP_ROTPLANE:
            o << "        float px = " << r(I.a) << ", py = " << r(I.a + 1) << ", pz = " << (D >= 3 ? r(I.a + 2) : "0.0f") << ";\n";
            if (D == 4) o << "        const float pw = " << r(I.a + 3) << ";\n";
            o << "        fnd::rotate_plane(" << I.aux << ", px, py, pz);\n";
            o << "        " << r(I.dst) << " = px; " << r(I.dst + 1) << " = py; " << r(I.dst + 2) << " = pz;\n";
            if (D == 4) o << "        " << r(I.dst + 3) << " = pw;\n";
            break;
        case FN_OP_NOISE: {
            o << "        const float f = " << p(0) << ";\n";
            if (const ColState* st = col ? col->at(pc) : nullptr) {
                o << "        " << r(I.dst) << " = fnd::scale_out(S.s" << pc << ".eval(tab[" << st->table << " + j]), " << p(1) << ", " << p(2)
                  << ", " << p(3) << ");\n";
                break;
            }
            o << "        " << r(I.dst) << " = fnd::scale_out(fnd::" << noise_fn(I.aux) << D << "(" << sd;
            for (int j = 0; j < D; ++j) o << ", " << r(I.a + j) << " * f";
            o << "), " << p(1) << ", " << p(2) << ", " << p(3) << ");\n";
            break;
        }
        case FN_OP_WHITE:
            o << "        const float pp[" << D << "] = " << pos(I.a) << ";\n";
            o << "        " << r(I.dst) << " = fnd::scale_out(fnd::white<" << D << ">(" << sd << ", pp), -fnd::kValueBounds, " << p(0) << ", " << p(1) << ");\n";
            break;
        case FN_OP_CHECKER:
            o << "        const float pp[" << D << "] = " << pos(I.a) << ";\n";
            o << "        " << r(I.dst) << " = fnd::scale_out(fnd::checkerboard<" << D << ">(pp, " << p(0) << "), 0.0f, " << p(1) << ", " << p(2) << ");\n";
            break;
        case FN_OP_SINE:
            o << "        const float pp[" << D << "] = " << pos(I.a) << ";\n";
            o << "        " << r(I.dst) << " = fnd::scale_out(fnd::sine_wave<" << D << ">(pp, " << p(0) << "), -1.0f, " << p(1) << ", " << p(2) << ");\n";
            break;
        case FN_OP_CELL_VALUE:
            o << "        const float pp[" << D << "] = " << pos(I.a) << ";\n        " << cellp(3) << "\n";
            o << "        " << r(I.dst) << " = fnd::scale_out(" << fast("value(") << "fnd::cellular_value<" << D << ">(" << sd << ", pp, cp, "
              << ((I.aux >> 4) & 3) << mk(I) << "), -fnd::kValueBounds, " << p(1) << ", " << p(2) << ");\n";
            break;
        case FN_OP_CELL_DIST:
            o << "        const float pp[" << D << "] = " << pos(I.a) << ";\n        " << cellp(3) << "\n";
            o << "        float dist[4];\n        ";
            if (cell) o << "if (" << cell_state << ".fast) " << cell_state << ".distances(" << cell_tab << ", dist); else ";
            o << "fnd::cellular_distances<" << D << ", "
              << std::max((I.aux >> 4) & 3, (I.aux >> 8) & 3) + 1 << ">(" << sd << ", pp, cp, dist" << mk(I) << ");\n";
            o << "        float nmax; const float v = fnd::cellular_return<" << D << ">(dist, cp.distFunc, " << ((I.aux >> 4) & 3) << ", "
              << ((I.aux >> 8) & 3) << ", " << ((I.aux >> 12) & 7) << ", nmax);\n";
            o << "        " << r(I.dst) << " = fnd::scale_out(v, 0.0f, " << p(1) << ", " << p(2) << ");\n";
            break;
        case FN_OP_CELL_LOOKUP:
            o << "        const float pp[" << D << "] = " << pos(I.a) << ";\n        " << cellp(2) << "\n";
            o << "        float oo[" << D << "];\n        ";
            if (cell) o << "if (" << cell_state << ".fast) " << cell_state << ".lookup(" << cell_tab << ", " << p(1) << ", oo); else ";
            o << "fnd::cellular_lookup_pos<" << D << ">(" << sd << ", pp, cp, " << p(1) << ", oo" << mk(I) << ");\n";
            for (int j = 0; j < D; ++j) o << "        " << r(I.dst + j) << " = oo[" << j << "];\n";
            break;
        case FN_OP_WARP_GRAD: case FN_OP_WARP_SIMPLEX:
            o << "        const float f = " << p(0) << ";\n";
            o << "        float sp[" << D << "], io[" << D << "];\n";
            for (int j = 0; j < D; ++j) o << "        sp[" << j << "] = " << r(I.a + j) << " * f; io[" << j << "] = " << r(I.dst + j) << ";\n";
            o << "        const float axis[" << D << "] = {";
            for (int j = 0; j < D; ++j) o << (j ? ", " : "") << p(1 + j);
            if (I.op == FN_OP_WARP_GRAD)
                o << "};\n        const float st = " << (cell ? cell_state + ".fast ? " + cell_state + ".warp(" + cell_tab + ", " + r(I.b) + ", axis, io) : " : std::string())
                  << "fnd::warp_gradient<" << D << ">(" << sd << ", " << r(I.b) << ", sp, axis, io);\n";
            else
                o << "};\n        const float st = fnd::warp_simplex<" << D << ">(" << sd << ", " << r(I.b) << ", sp, axis, io, "
                  << ((I.aux & 1) ? "true" : "false") << ", " << ((I.aux & 2) ? "true" : "false") << ");\n";
            for (int j = 0; j < D; ++j) o << "        " << r(I.dst + j) << " = io[" << j << "];\n";
            if (I.c != FN_REG_NONE) o << "        " << r(I.c) << " = st;\n";
            else o << "        (void)st;\n";
            break;
        case FN_OP_FRACT_INIT:
            if (I.aux) o << "        const float nz = fnd::fabs_(" << r(I.a) << "); " << r(I.a) << " = nz; " << r(I.dst) << " = (nz * -2.0f + 1.0f) * 1.0f;\n";
            else o << "        " << r(I.dst) << " = " << r(I.a) << " * 1.0f;\n";
            o << "        " << r(I.b) << " = 1.0f;\n";
            break;
        case FN_OP_FRACT_AMP:
            if (is_zero(I.c) && known[I.a].what == kBounded) {
                o << "        " << r(I.b) << " = " << r(I.b) << " * " << r(I.d) << ";\n";
                break;
            }
            o << "        const float t = " << (I.aux ? "1.0f - " + r(I.a) : "(" + r(I.a) + " + 1.0f) * 0.5f") << ";\n";
            o << "        const float amp = " << r(I.b) << " * fnd::lerp(1.0f, t, " << r(I.c) << ");\n";
            o << "        " << r(I.b) << " = amp * " << r(I.d) << ";\n";
            break;
        case FN_OP_FRACT_ACC:
            if (I.aux) o << "        const float nz = fnd::fabs_(" << r(I.a) << "); " << r(I.a) << " = nz; " << r(I.dst) << " = " << r(I.dst) << " + (nz * -2.0f + 1.0f) * " << r(I.b) << ";\n";
            else o << "        " << r(I.dst) << " = " << r(I.dst) << " + " << r(I.a) << " * " << r(I.b) << ";\n";
            break;
        case FN_OP_DWF_AMP:
            if (is_zero(I.c) && known[I.a].what == kWarpStrength) {
                o << "        " << r(I.b) << " = " << r(I.b) << " * " << r(I.d) << ";\n";
                break;
            }
            o << "        const float s = sqrtf(" << r(I.a) << "); " << r(I.a) << " = s;\n";
            o << "        const float amp = " << r(I.b) << " * fnd::lerp(1.0f, 1.0f - s, " << r(I.c) << ");\n";
            o << "        " << r(I.b) << " = amp * " << r(I.d) << ";\n";
            break;
        case FN_OP_ADD: o << "        " << r(I.dst) << " = " << r(I.a) << " + " << r(I.b) << ";\n"; break;
        case FN_OP_SUB: o << "        " << r(I.dst) << " = " << r(I.a) << " - " << r(I.b) << ";\n"; break;
        case FN_OP_MUL: o << "        " << r(I.dst) << " = " << r(I.a) << " * " << r(I.b) << ";\n"; break;
        case FN_OP_DIV: o << "        " << r(I.dst) << " = " << r(I.a) << " / " << r(I.b) << ";\n"; break;
        case FN_OP_MOD: o << "        " << r(I.dst) << " = fnd::mod_(" << r(I.a) << ", " << r(I.b) << ");\n"; break;
        case FN_OP_MIN: o << "        " << r(I.dst) << " = fnd::fmin_(" << r(I.a) << ", " << r(I.b) << ");\n"; break;
        case FN_OP_MAX: o << "        " << r(I.dst) << " = fnd::fmax_(" << r(I.a) << ", " << r(I.b) << ");\n"; break;
        case FN_OP_ABS: o << "        " << r(I.dst) << " = fnd::fabs_(" << r(I.a) << ");\n"; break;
        case FN_OP_SSQRT: o << "        " << r(I.dst) << " = fnd::signed_sqrt(" << r(I.a) << ");\n"; break;
        case FN_OP_POWF: o << "        " << r(I.dst) << " = fnd::pow_(fnd::fmax_(fnd::fabs_(" << r(I.a) << "), 1.17549435e-38f), " << r(I.b) << ");\n"; break;
        case FN_OP_POWI:
            o << "        const float v = " << r(I.a) << "; float pw = v * v;\n";
            o << "        for (int i = 2; i < " << I.aux << "; ++i) pw *= v;\n        " << r(I.dst) << " = pw;\n";
            break;
        case FN_OP_MINSMOOTH: o << "        " << r(I.dst) << " = fnd::min_smooth(" << r(I.a) << ", " << r(I.b) << ", " << r(I.c) << ");\n"; break;
        case FN_OP_MAXSMOOTH: o << "        " << r(I.dst) << " = -fnd::min_smooth(-" << r(I.a) << ", -" << r(I.b) << ", " << r(I.c) << ");\n"; break;
        case FN_OP_FADE:
            o << "        " << r(I.dst) << " = fnd::lerp(" << r(I.a) << ", " << r(I.b) << ", fnd::fade_t(" << r(I.c) << ", " << r(I.d) << ", " << r(I.e)
              << ", " << I.aux << "));\n";
            break;
        case FN_OP_REMAP:
            o << "        " << r(I.dst) << " = fnd::remap(" << r(I.a) << ", " << r(I.b) << ", " << r(I.c) << ", " << r(I.d) << ", " << r(I.e) << ", "
              << (I.aux ? "true" : "false") << ");\n";
            break;
        case FN_OP_TERRACE:
            o << "        const float src = " << r(I.a) << " * " << p(0) << ";\n        float rounded = rintf(src);\n";
            if (I.b != FN_REG_NONE)
                o << "        const float sm = " << r(I.b) << ";\n        if (sm != 0.0f) rounded = fnd::terrace_smooth(rounded, src, 1.0f + 1.0f / sm);\n";
            else if (I.aux)
                o << "        rounded = fnd::terrace_smooth(rounded, src, " << p(2) << ");\n";
            o << "        " << r(I.dst) << " = rounded * " << p(1) << ";\n";
            break;
        case FN_OP_PINGPONG: o << "        " << r(I.dst) << " = fnd::ping_pong(" << r(I.a) << " * " << r(I.b) << ");\n"; break;
        case FN_OP_RGBA8: o << "        " << r(I.dst) << " = fnd::to_rgba8(" << r(I.a) << ", " << p(0) << ", " << p(1) << ");\n"; break;
        case FN_OP_GRADIENT: {
            const int off[4] = {I.b, I.c, I.d, I.e};
            o << "        float acc = 0.0f;\n";
            for (int j = 0; j < D; ++j) o << "        acc = fmaf(" << r(I.a + j) << " + " << r(off[j]) << ", " << p(j) << ", acc);\n";
            o << "        " << r(I.dst) << " = acc;\n";
            break;
        }
        case FN_OP_DISTANCE:
            o << "        const float pp[" << D << "] = " << pos(I.a) << ";\n";
            o << "        " << r(I.dst) << " = fnd::distance<" << D << ">(" << (I.aux & 15) << ", " << (((I.aux >> 4) & 1) ? "true" : "false")
              << ", pp, " << (I.b != FN_REG_NONE ? r(I.b) : std::string("0.0f")) << ");\n";
            break;
        default:
            o << "        // unsupported op\n";
            break;
        }
        o << "    }\n";
        switch (I.op) {
        case FN_OP_MOV: known[I.dst] = known[I.a]; break;
        case FN_OP_CONST: known[I.dst].what = kConst; known[I.dst].value = P[I.prm]; break;
        case FN_OP_NOISE: {
            const bool bounded = std::fabs(P[I.prm + 1]) * std::fabs(P[I.prm + 2]) < 1e30f && std::fabs(P[I.prm + 3]) < 1e30f;
            known[I.dst].what = bounded ? kBounded : kUnknown;
            break;
        }
        case FN_OP_FRACT_INIT: case FN_OP_FRACT_ACC: known[I.dst].what = known[I.b].what = kUnknown; break;   // a keeps its size (abs)
        case FN_OP_FRACT_AMP: known[I.b].what = kUnknown; break;
        case FN_OP_DWF_AMP: known[I.a].what = known[I.b].what = kUnknown; break;
        default:
            for (int j = 0; j < 4; ++j) known[I.dst + j].what = kUnknown;
            if ((I.op == FN_OP_WARP_GRAD || I.op == FN_OP_WARP_SIMPLEX) && I.c != FN_REG_NONE)
                known[I.c].what = I.op == FN_OP_WARP_GRAD ? kWarpStrength : kUnknown;
            break;
        }
    }
    o << "    return " << r(h->out_reg) << ";\n}\n\n";
}

// Unit `u` of a column launch: 32 neighbouring points of the grid's plane (all axes but the
// last; one per lane, lanes past the plane repeat its last point and store nothing), walked
// along the last axis for up to A.col_len steps.
void emit_column_unit(const CompiledProgram& prog, const std::string& eval, const std::string& name, std::ostringstream& o)
{
    const int D = prog.dim;
    const char* pv[4] = {"px", "py", "pz", "pw"};
    const std::string fixed = std::string("px, ") + (D > 2 ? "py" : "0.0f") + ", " + (D > 3 ? "pz" : "0.0f");
    o << "__device__ __forceinline__ void " << name << "(const fn::PointArgs& A, float* __restrict__ out, unsigned u, float4* tab, float& mn, float& mx)\n{\n"
      << "    const unsigned plane = A.col_plane, chunks = (plane + 31u) >> 5;\n"
      << "    const unsigned seg = u / chunks, p = (u - seg * chunks) * 32u + (threadIdx.x & 31u);\n"
      << "    const bool live = p < plane;\n"
      << "    unsigned r = live ? p : plane - 1u;\n";
    for (int j = 0; j < D - 1; ++j) {
        if (j < D - 2)
            o << "    const unsigned q" << j << " = fne::fast_div(r, A.divm[" << j << "], A.divs[" << j << "]);\n"
              << "    const float " << pv[j] << " = fmaf(fnd::cvtf((int)(r - q" << j << " * (unsigned)A.count[" << j << "])), A.step[" << j
              << "], A.offset[" << j << "]); r = q" << j << ";\n";
        else
            o << "    const float " << pv[j] << " = fmaf(fnd::cvtf((int)r), A.step[" << j << "], A.offset[" << j << "]);\n";
    }
    o << "    const unsigned t0 = seg * A.col_len, t1 = A.col_steps - t0 < A.col_len ? A.col_steps : t0 + A.col_len;\n"
      << "    float* dst = out + (unsigned long long)t0 * plane + p;\n"
      << "    const unsigned lane = threadIdx.x & 31u;\n"
      << "    " << eval << "_state S;\n    S.init(" << fixed << ");\n"
      << "#pragma unroll 1\n"
      << "    for (unsigned tb = t0; tb < t1; tb += 32u) {\n"
      << "        const unsigned fresh = S.prepare(tab, lane, fmaf(fnd::cvtf((int)(A.col_first + tb + lane)), A.step[" << D - 1
      << "], A.offset[" << D - 1 << "]));\n"
      << "        __syncwarp();\n"
      << "        const unsigned n = t1 - tb < 32u ? t1 - tb : 32u;\n"
      << "        fne::wait_for_stream();\n"
      << "        for (unsigned j = 0; j < n;) {\n"
      << "            if ((fresh >> j) & 1u) S.enter(A.seed, tab, j, " << fixed << ");\n"
      << "            const unsigned ahead = (fresh >> j) >> 1, run = ahead ? j + (unsigned)__ffs((int)ahead) : n, stop = run < n ? run : n;\n"
      << "#pragma unroll 1\n"
      << "            for (; j < stop; ++j, dst += plane) {\n"
      << "                const float " << pv[D - 1] << " = fmaf(fnd::cvtf((int)(A.col_first + tb + j)), A.step[" << D - 1 << "], A.offset[" << D - 1 << "]);\n"
      << "                const float v = " << eval << "(A.seed";
    for (int j = 0; j < 4; ++j) o << ", " << (j < D ? pv[j] : "0.0f");
    o << ", S, tab, j);\n"
      << "                if (live) *dst = v;\n"
      << "                fne::fold(v, mn, mx);\n"
      << "            }\n"
      << "        }\n"
      << "        __syncwarp();\n"
      << "    }\n}\n\n";
}

// 256-thread blocks per SM a column kernel is bounded to, by the registers its state holds
// beside the ~25-60 the step itself needs.  Keeping every state is worth more than warps:
// FBm(Perlin) 4D 32^4 takes 23 us with five octaves' states and one block, 37 us with four, 54 us
// with two octaves' and two blocks; FBm(Perlin) 256^3 (100 registers of state) 142 us with two
// blocks, 156 with one, 243 with three (spills); terrain and CellularLookup 160^3 (31 registers)
// 269 and 55 us with two blocks, 279 and 60 with three, 290 and 66 with four; terrain 2048^2 (17
// registers) 105 us with four, 109 with two.
int column_blocks(const ColPlan& plan) { return plan.regs <= 20 ? 4 : plan.regs <= 104 ? 2 : 1; }

// The per-call kernel that walks a grid in columns.
void emit_percall_column(const CompiledProgram& prog, const ColPlan& plan, std::ostringstream& o)
{
    emit_column_unit(prog, "fnjit_ceval_0", "fnjit_colunit_0", o);
    o << "extern \"C\" __global__ void __launch_bounds__(256, " << column_blocks(plan) << ") fnjit_col_0"
      << "(fn::PointArgs A, float* __restrict__ out, fn::MinMaxWork* work, float* dminmax, unsigned early)\n{\n"
      << "    __shared__ float4 tab[8][" << plan.table << "];\n"
      << "    __shared__ float smn[8], smx[8];\n"
      << "    if (early) fne::let_stream_continue();\n"
      << gradient_setup(prog, &plan)
      << "    float mn = fne::inf(), mx = -fne::inf();\n"
      << "    for (unsigned u = blockIdx.x * 8u + (threadIdx.x >> 5); u < A.col_units; u += gridDim.x * 8u)\n"
      << "        fnjit_colunit_0(A, out, u, tab[threadIdx.x >> 5], mn, mx);\n"
      << "    fne::let_stream_continue();\n"
      << "    fne::grid_minmax(mn, mx, work, dminmax, smn, smx);\n"
      << "}\n\n";
}

// Per-call kernels for program k: grid / position array / tileable.
//
// Each warp owns chunks of 32*ppl consecutive points (ppl = points per lane,
// 1..4, chosen by the host).  Lane l evaluates points chunk + 32*t + l
// (t < ppl, one point at a time, so the tree's code is not replicated) and
// parks the values in shared memory; with ppl == 4 the warp then writes the
// chunk as 32 float4 stores (512 contiguous bytes per warp).  Small calls use
// ppl == 1 so that their few points spread over as many SMs as possible.
enum PercallKernels : unsigned { kGridKernel = 1, kPositionKernel = 2, kOtherKernels = 4 };
void emit_percall(const CompiledProgram& prog, int k, unsigned which, std::ostringstream& o)
{
    const int D = prog.dim;
    const char* pv[4] = {"px", "py", "pz", "pw"};
    std::string call = "fnjit_eval_" + std::to_string(k) + "(A.seed";
    for (int j = 0; j < 4; ++j) call += std::string(", ") + (j < D ? pv[j] : "0.0f");
    call += ")";

    auto kernel = [&](const char* name, const std::string& prologue, const std::string& position) {
        // prologue: before the first point (a kernel that reads the caller's arrays waits there).  See
        // begin_early for early.
        const bool waits = !prologue.empty();
        o << "extern \"C\" __global__ void __launch_bounds__(256, 4) " << name << "_" << k
          << "(fn::PointArgs A, float* __restrict__ out, fn::MinMaxWork* work, float* dminmax, unsigned ppl, unsigned early)\n{\n"
          << "    __shared__ float4 stage[8][32];\n"
          << "    __shared__ float smn[8], smx[8];\n"
          << (waits ? "    if (early) fne::let_stream_continue();\n" : "    fne::let_stream_continue();\n")
          << gradient_setup(prog)
          << "    float mn = fne::inf(), mx = -fne::inf();\n"
          << "    const unsigned total = (unsigned)A.total;\n"
          << "    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;\n"
          << "    const unsigned nwarps = (gridDim.x * blockDim.x) >> 5;\n"
          << "    const bool aligned = (((unsigned long long)out) & 15ull) == 0;\n"
          << "    float* st = reinterpret_cast<float*>(stage[warp]);\n"
          << prologue
          << "    const unsigned chunk = 32u * ppl;\n"
          << "    for (unsigned base = (((blockIdx.x * blockDim.x) >> 5) + warp) * chunk; base < total; base += nwarps * chunk) {\n"
          << "#pragma unroll 1\n"
          << "        for (unsigned t = 0; t < ppl; ++t) {\n"
          << "            const unsigned i = base + t * 32u + lane;\n"
          << "            float v = 0.0f;\n"
          << "            if (i < total) {\n"
          << position
          << "                v = " << call << ";\n"
          << "                fne::fold(v, mn, mx);\n"
          << "            }\n"
          << "            st[t * 32u + lane] = v;\n"
          << "        }\n"
          << "        __syncwarp();\n"
          << "        fne::wait_for_stream();\n"
          << "        if (ppl == 4u && aligned && base + 128u <= total) {\n"
          << "            reinterpret_cast<float4*>(out + base)[lane] = stage[warp][lane];\n"
          << "        } else {\n"
          << "            for (unsigned q = 0; q < ppl; ++q) {\n"
          << "                const unsigned j = base + q * 32u + lane;\n"
          << "                if (j < total) out[j] = st[q * 32u + lane];\n"
          << "            }\n"
          << "        }\n"
          << "        __syncwarp();\n"
          << "    }\n"
          << (waits ? "    fne::let_stream_continue();\n" : "")
          << "    fne::grid_minmax(mn, mx, work, dminmax, smn, smx);\n"
          << "}\n\n";
    };

    // grid: Generator.inl:79-254, pos_k = fma(float(i_k), step_k, offset_k), x fastest
    std::string gridpos;
    {
        std::ostringstream pos;
        pos << "                unsigned r = i + A.base;\n";          // index in the whole request
        const char* ax = "xyzw";
        for (int j = 0; j < D; ++j) {
            if (j < D - 1)
                pos << "                const unsigned q" << j << " = fne::fast_div(r, A.divm[" << j << "], A.divs[" << j << "]);\n"
                    << "                const unsigned i" << ax[j] << " = r - q" << j << " * (unsigned)A.count[" << j << "]; r = q" << j << ";\n";
            else pos << "                const unsigned i" << ax[j] << " = r;\n";
            pos << "                const float " << pv[j] << " = fmaf(fnd::cvtf((int)i" << ax[j] << "), A.step[" << j << "], A.offset[" << j << "]);\n";
        }
        gridpos = pos.str();
        if (which & kGridKernel) kernel("fnjit_grid", "", gridpos);
    }
    // position arrays: Generator.inl:256-350, pos_k = offset_k + array_k[i].  Plain loads: the arrays
    // may be written while this kernel already waits, so they are not read-only to it.
    if (which & kPositionKernel) {
        std::ostringstream pos;
        for (int j = 0; j < D; ++j)
            pos << "                const float " << pv[j] << " = A.offset[" << j << "] + A.pos[" << j << "][i + A.base];\n";
        kernel("fnjit_pos", "    fne::wait_for_stream();\n", pos.str());
    }
    // tileable (4D programs): Generator.inl:370-433
    if (D == 4 && (which & kOtherKernels)) {
        std::ostringstream pos;
        pos << "                const unsigned g = i + A.base;\n"
            << "                const unsigned iy = fne::fast_div(g, A.divm[0], A.divs[0]), ix = g - iy * (unsigned)A.count[0];\n"
            << "                const float xf = fnd::cvtf((int)ix) * A.tmul[0];\n"
            << "                const float yf = fnd::cvtf((int)iy) * A.tmul[1];\n"
            << "                const float px = fnd::cos_(xf) * A.tfreq[0];\n"
            << "                const float py = fnd::cos_(yf) * A.tfreq[1];\n"
            << "                const float pz = fnd::sin_(xf) * A.tfreq[0];\n"
            << "                const float pw = fnd::sin_(yf) * A.tfreq[1];\n";
        kernel("fnjit_tile", "", pos.str());
    }
    // Chunk meshing (3D programs): the meshers need every density only as "above the iso
    // level" / "at or below it", and exact values at a few voxels near the surface.
    //  fnjit_solid: the grid's two classification bitmasks (bit i of word i / 32; the warp's
    //    32 consecutive points form one word) and OutputMinMax -- no density leaves registers;
    //  fnjit_list: the grid's values at listed point indices (count read from the device).
    if (D == 3 && (which & kOtherKernels)) {
        o << "extern \"C\" __global__ void __launch_bounds__(256, 4) fnjit_solid_" << k
          << "(fn::PointArgs A, unsigned* __restrict__ above, unsigned* __restrict__ solid, fn::MinMaxWork* work, float* dminmax,\n"
          << "    float iso, unsigned ppl)\n{\n"
          << "    __shared__ float smn[8], smx[8];\n"
          << gradient_setup(prog)
          << "    float mn = fne::inf(), mx = -fne::inf();\n"
          << "    const unsigned total = (unsigned)A.total;\n"
          << "    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;\n"
          << "    const unsigned nwarps = (gridDim.x * blockDim.x) >> 5;\n"
          << "    const unsigned chunk = 32u * ppl;\n"
          << "    for (unsigned base = (((blockIdx.x * blockDim.x) >> 5) + warp) * chunk; base < total; base += nwarps * chunk) {\n"
          << "#pragma unroll 1\n"
          << "        for (unsigned t = 0; t < ppl; ++t) {\n"
          << "            const unsigned i = base + t * 32u + lane;\n"
          << "            bool gt = false, le = false;\n"
          << "            if (i < total) {\n"
          << gridpos
          << "                const float v = " << call << ";\n"
          << "                fne::fold(v, mn, mx);\n"
          << "                gt = v > iso;\n"
          << "                le = v <= iso;\n"
          << "            }\n"
          << "            const unsigned wg = __ballot_sync(0xffffffffu, gt), wl = __ballot_sync(0xffffffffu, le);\n"
          << "            if (lane == 0 && base + t * 32u < total) { above[(base + t * 32u) >> 5] = wg; solid[(base + t * 32u) >> 5] = wl; }\n"
          << "        }\n"
          << "    }\n"
          << "    fne::grid_minmax(mn, mx, work, dminmax, smn, smx);\n"
          << "}\n\n";
        o << "extern \"C\" __global__ void __launch_bounds__(256, 4) fnjit_list_" << k
          << "(fn::PointArgs A, const unsigned* __restrict__ idx, const unsigned* __restrict__ count, float* __restrict__ out)\n{\n"
          << gradient_setup(prog)
          << "    const unsigned n = *count;\n"
          << "    for (unsigned j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {\n"
          << "        const unsigned i = idx[j];\n"
          << gridpos
          << "        out[j] = " << call << ";\n"
          << "    }\n"
          << "}\n\n";
    }
}

}  // namespace

const std::vector<BatchVariant>& batch_variants()
{
    // {threads, register bound as blocks per SM, points per thread per loop iteration}
    static const std::vector<BatchVariant> v = {
        {256, 4, 1},     // 64 registers: the kernel fnJitCompile builds
        {256, 3, 1},     // 80 registers: fewer spills for long cellular walks
        {256, 2, 1},     // 128 registers
        {128, 8, 1},     // 64 registers in smaller blocks: finer balance of the work queue
        {256, 2, 2},     // 128 registers, two points in flight per thread
    };
    return v;
}

namespace {

std::string batch_kernel_name(size_t k, int variant)
{
    return "fnjit_batch_" + std::to_string(k) + (variant ? "_v" + std::to_string(variant) : std::string());
}

// The batch kernels: persistent CTAs pull (request, tile) items of their tree's
// group and run a tile loop with that tree's code inlined.  A variant fixes the
// block size, the register bound and how many points a thread has in flight.
void emit_batch(const std::vector<const CompiledProgram*>& progs, std::ostringstream& o, int variant)
{
    const BatchVariant bv = batch_variants()[(size_t)variant];
    for (size_t k = 0; k < progs.size(); ++k) {
        const int D = progs[k]->dim;
        const std::string call = "fnjit_eval_" + std::to_string(k) + "(A.seed, p[0], p[1], " + (D > 2 ? "p[2]" : "0.0f") +
                                 ", " + (D > 3 ? "p[3]" : "0.0f") + ")";
        o << "__device__ __forceinline__ void fnjit_tile_" << k << "_v" << variant
          << "(const fn::PointArgs& A, float* __restrict__ out, unsigned i, unsigned end, float& mn, float& mx)\n{\n";
        if (bv.points == 1) {
            o << "    for (; i < end; i += blockDim.x) {\n"
              << "        float p[4];\n"
              << "        fne::root_position32<" << D << ">(A, i, p);\n"
              << "        const float v = " << call << ";\n"
              << "        out[i] = v;\n"
              << "        fne::fold(v, mn, mx);\n"
              << "    }\n}\n\n";
        } else {
            o << "    for (; i < end; i += " << bv.points << "u * blockDim.x) {\n"
              << "        float v[" << bv.points << "];\n"
              << "#pragma unroll\n"
              << "        for (int q = 0; q < " << bv.points << "; ++q) {\n"
              << "            const unsigned j = i + q * blockDim.x;\n"
              << "            float p[4];\n"
              << "            fne::root_position32<" << D << ">(A, j < end ? j : i, p);\n"
              << "            v[q] = " << call << ";\n"
              << "        }\n"
              << "#pragma unroll\n"
              << "        for (int q = 0; q < " << bv.points << "; ++q) {\n"
              << "            const unsigned j = i + q * blockDim.x;\n"
              << "            if (j < end) { out[j] = v[q]; fne::fold(v[q], mn, mx); }\n"
              << "        }\n"
              << "    }\n}\n\n";
        }
    }
    // one persistent kernel per tree: each gets the register allocation its own
    // code needs, and the trees of a batch run as concurrent kernels
    for (size_t k = 0; k < progs.size(); ++k) {
        o << "extern \"C\" __global__ void __launch_bounds__(" << bv.threads << ", " << bv.min_blocks << ") "
          << batch_kernel_name(k, variant)
          << "(fn::BatchHeader* hdr, const fn::BatchRequest* __restrict__ reqs, fn::BatchState* states,\n"
             "    const uint2* __restrict__ items, fn::BatchGroup* grp)\n{\n"
             "    __shared__ unsigned int s_item;\n"
             "    __shared__ float smn[" << bv.threads / 32 << "], smx[" << bv.threads / 32 << "];\n"
          << gradient_setup(*progs[k]) <<
             "    const unsigned int first = grp->item_begin, last = grp->item_end;\n"
             "    const unsigned int tile_points = hdr->tile_points;\n"
             "    for (;;) {\n"
             "        if (threadIdx.x == 0) s_item = first + atomicAdd(&grp->head, 1u);\n"
             "        __syncthreads();\n"
             "        const unsigned int it = s_item;\n"
             "        __syncthreads();\n"
             "        if (it >= last) break;\n"
             "        const uint2 item = items[it];\n"
             "        const fn::BatchRequest& rq = reqs[item.x];\n"
             "        const fn::PointArgs args = rq.args;\n"
             "        const unsigned total = (unsigned)args.total;\n"
             "        const unsigned begin = item.y * tile_points;\n"
             "        const unsigned end = total - begin < tile_points ? total : begin + tile_points;\n"
             "        float mn = fne::inf(), mx = -fne::inf();\n"
             "        fnjit_tile_" << k << "_v" << variant << "(args, rq.out, begin + threadIdx.x, end, mn, mx);\n"
             "        fne::block_minmax(mn, mx, smn, smx);\n"
             "        if (threadIdx.x == 0) fne::finish_tile(rq, states + item.x, hdr, mn, mx);\n"
             "    }\n}\n\n";
    }
}

// The batch kernel of a tree's grid requests walked in columns: a work item is eight
// consecutive units of one request, one per warp.
void emit_batch_column(const CompiledProgram& prog, size_t k, const ColPlan& plan, std::ostringstream& o)
{
    const std::string id = std::to_string(k);
    emit_column_unit(prog, "fnjit_ceval_" + id, "fnjit_colunit_" + id, o);
    o << "extern \"C\" __global__ void __launch_bounds__(256, " << column_blocks(plan) << ") fnjit_bcol_" << id
      << "(fn::BatchHeader* hdr, const fn::BatchRequest* __restrict__ reqs, fn::BatchState* states,\n"
         "    const uint2* __restrict__ items, fn::BatchGroup* grp)\n{\n"
         "    __shared__ float4 tab[8][" << plan.table << "];\n"
         "    __shared__ unsigned int s_item;\n"
         "    __shared__ float smn[8], smx[8];\n"
      << gradient_setup(prog, &plan) <<
         "    const unsigned int first = grp->item_begin, last = grp->item_end;\n"
         "    for (;;) {\n"
         "        if (threadIdx.x == 0) s_item = first + atomicAdd(&grp->head, 1u);\n"
         "        __syncthreads();\n"
         "        const unsigned int it = s_item;\n"
         "        __syncthreads();\n"
         "        if (it >= last) break;\n"
         "        const uint2 item = items[it];\n"
         "        const fn::BatchRequest& rq = reqs[item.x];\n"
         "        const fn::PointArgs args = rq.args;\n"
         "        const unsigned u = item.y * 8u + (threadIdx.x >> 5);\n"
         "        float mn = fne::inf(), mx = -fne::inf();\n"
         "        if (u < args.col_units) fnjit_colunit_" << id << "(args, rq.out, u, tab[threadIdx.x >> 5], mn, mx);\n"
         "        fne::block_minmax(mn, mx, smn, smx);\n"
         "        if (threadIdx.x == 0) fne::finish_tile(rq, states + item.x, hdr, mn, mx);\n"
         "    }\n}\n\n";
}

// A module's loaded programs.
struct Module {
    std::vector<cudaLibrary_t> parts;
    Module() = default;
    Module(const Module&) = delete;
    Module& operator=(const Module&) = delete;
    ~Module()
    {
        for (cudaLibrary_t lib : parts) cudaLibraryUnload(lib);
    }
};

std::mutex g_jit_mu;
std::unordered_map<uint64_t, JitKernels> g_kernels;
std::vector<std::unique_ptr<Module>>& g_modules = *new std::vector<std::unique_ptr<Module>>;   // never unloaded
std::unordered_map<uint64_t, cudaKernel_t> g_batch_kernels;   // per-tree batch kernel (variant 0)
std::unordered_map<uint64_t, std::vector<BatchKernel>> g_batch_variant_kernels;   // per tree: every variant built
std::atomic<bool> g_enabled{true};

}  // namespace

namespace {

// What NVRTC takes for a kernel that evaluates `prog` once, beyond the module's head (seconds on a
// Grace core, roughly: FBm(Perlin) 3D 0.13, 4D 0.9, terrain 3D 0.27).
float compile_seconds(const CompiledProgram& prog)
{
    const FnProgramHeader* h = reinterpret_cast<const FnProgramHeader*>(prog.blob.data());
    const FnInstr* ins = fn_program_instrs(h);
    static const float simplex[3] = {7, 14, 21}, super[3] = {14, 35, 40}, perlin[3] = {8, 26, 180}, value[3] = {7, 14, 28}, warp[3] = {7, 14, 35},
                       cells[3] = {28, 56, 56};
    float ms = 0;
    for (int pc = 0; pc < h->n_instr; ++pc) {
        const FnInstr& I = ins[pc];
        const int d = I.dim - 2;
        switch (I.op) {
        case FN_OP_NOISE: ms += (I.aux == FN_NOISE_SIMPLEX ? simplex : I.aux == FN_NOISE_SUPERSIMPLEX ? super : I.aux == FN_NOISE_PERLIN ? perlin : value)[d]; break;
        case FN_OP_WARP_GRAD: ms += warp[d]; break;
        case FN_OP_WARP_SIMPLEX: ms += 3 * warp[d]; break;
        case FN_OP_CELL_VALUE: case FN_OP_CELL_DIST: case FN_OP_CELL_LOOKUP: ms += cells[d]; break;
        default: ms += 0.5f; break;
        }
    }
    for (auto& sub : prog.subs) ms += 1e3f * compile_seconds(sub);
    return 1e-3f * ms;
}

std::string module_head(const std::string& what)
{
    return "// generated by fn_jit.cpp: " + what + "\n#define FN_GRADIENT_TABLE\n" + embedded_device_source() + "\n";
}

}  // namespace

ModuleSource jit_batch_module(const std::vector<const CompiledProgram*>& progs, int variant)
{
    std::ostringstream o;
    for (size_t k = 0; k < progs.size(); ++k) emit_eval(*progs[k], "fnjit_eval_" + std::to_string(k), o);
    emit_batch(progs, o, variant);
    float seconds = 0;
    for (auto* p : progs) seconds += compile_seconds(*p);
    ModuleSource m{module_head("batch module, variant " + std::to_string(variant)), {{o.str(), seconds}}};
    for (size_t k = 0; variant == 0 && k < progs.size(); ++k) {
        const ColPlan plan = column_plan(*progs[k]);
        if (plan.states.empty()) continue;
        std::ostringstream c;
        emit_eval(*progs[k], "fnjit_ceval_" + std::to_string(k), c, &plan);
        emit_batch_column(*progs[k], k, plan, c);
        m.parts.push_back({c.str(), compile_seconds(*progs[k])});
    }
    return m;
}

ModuleSource jit_percall_module(const CompiledProgram& prog)
{
    const ColPlan plan = column_plan(prog);
    std::ostringstream eval;
    emit_eval(prog, "fnjit_eval_0", eval);
    ModuleSource m{module_head("per-call module") + eval.str(), {}};
    for (unsigned which : {(unsigned)kGridKernel, (unsigned)kPositionKernel, (unsigned)kOtherKernels}) {
        std::ostringstream o;
        emit_percall(prog, 0, which, o);
        if (!o.str().empty()) m.parts.push_back({o.str(), (which == kOtherKernels && prog.dim == 3 ? 2.0f : 1.0f) * compile_seconds(prog)});
    }
    if (!plan.states.empty()) {
        std::ostringstream c;
        emit_eval(prog, "fnjit_ceval_0", c, &plan);
        emit_percall_column(prog, plan, c);
        m.parts.push_back({c.str(), compile_seconds(prog)});
    }
    return m;
}

// ---------------------------------------------------------------- on-disk module cache
// Compiled modules are kept on disk, keyed by their CUDA source (which embeds the node
// library's device code), the NVRTC options and the NVRTC version, so a module that any
// earlier process built loads in milliseconds instead of being compiled again.  File:
// "FNJC", format version, the 128-bit key, payload size, the module (its cubins, see
// pack_parts), a checksum of it; a file that does not check out is ignored (and replaced by the
// next compile).
namespace {

constexpr uint32_t kCacheFormat = 2;
const char* const kNvrtcOptions[] = {"--gpu-architecture=sm_103a", "-fmad=false", "--std=c++17", "-default-device",
                                     "-lineinfo", "-diag-suppress=177"};

struct CacheKey {
    uint64_t a = 0, b = 0;
};

uint64_t fnv1a(const void* data, size_t n, uint64_t h)
{
    const unsigned char* p = static_cast<const unsigned char*>(data);
    for (size_t i = 0; i < n; ++i) h = (h ^ p[i]) * 0x100000001B3ull;
    return h;
}

CacheKey cache_key(const ModuleSource& src)
{
    int major = 0, minor = 0;
    nvrtcVersion(&major, &minor);
    std::string salt = "nvrtc " + std::to_string(major) + "." + std::to_string(minor) + " format " + std::to_string(kCacheFormat);
    for (const char* o : kNvrtcOptions) salt += std::string(" ") + o;
    CacheKey k;
    k.a = fnv1a(salt.data(), salt.size(), 0xCBF29CE484222325ull);
    k.b = fnv1a(salt.data(), salt.size(), 0x84222325CBF29CE4ull ^ 0x9E3779B97F4A7C15ull);
    auto add = [&](const std::string& text) {
        k.a = fnv1a(text.data(), text.size(), k.a);
        k.b = fnv1a(text.data(), text.size(), k.b);
    };
    add(src.head);
    for (const ModuleSource::Part& part : src.parts) add(part.text);
    return k;
}

std::mutex g_cache_mu;
bool g_cache_resolved = false;
std::string g_cache_dir;                  // empty: off
std::atomic<unsigned long long> g_cache_hits{0}, g_cache_misses{0};

void make_dirs(const std::string& dir)
{
    for (size_t i = 1; i <= dir.size(); ++i)
        if (i == dir.size() || dir[i] == '/') mkdir(dir.substr(0, i).c_str(), 0755);   // existing parts fail harmlessly
}

std::string cache_dir()
{
    std::lock_guard<std::mutex> lk(g_cache_mu);
    if (!g_cache_resolved) {
        g_cache_resolved = true;
        // off unless the application names a directory: a library writes no files of its own
        const char* env = std::getenv("FASTNOISE_JIT_CACHE");
        if (env && *env && std::strcmp(env, "off") != 0) g_cache_dir = env;
        if (!g_cache_dir.empty()) make_dirs(g_cache_dir);
    }
    return g_cache_dir;
}

std::string cache_path(const std::string& dir, const CacheKey& k)
{
    char name[64];
    std::snprintf(name, sizeof name, "/%016llx%016llx.cubin", (unsigned long long)k.a, (unsigned long long)k.b);
    return dir + name;
}

bool cache_read(const std::string& path, const CacheKey& k, std::vector<char>& cubin)
{
    std::ifstream f(path, std::ios::binary);
    if (!f) return false;
    char magic[4];
    uint32_t format = 0;
    uint64_t ka = 0, kb = 0, size = 0, sum = 0;
    if (!f.read(magic, 4) || std::memcmp(magic, "FNJC", 4) != 0 || !f.read(reinterpret_cast<char*>(&format), 4) ||
        format != kCacheFormat || !f.read(reinterpret_cast<char*>(&ka), 8) || !f.read(reinterpret_cast<char*>(&kb), 8) ||
        ka != k.a || kb != k.b || !f.read(reinterpret_cast<char*>(&size), 8) || size == 0 || size > (uint64_t(1) << 30))
        return false;
    std::vector<char> data((size_t)size);
    if (!f.read(data.data(), (std::streamsize)size) || !f.read(reinterpret_cast<char*>(&sum), 8) ||
        sum != fnv1a(data.data(), data.size(), 0xCBF29CE484222325ull))
        return false;
    cubin.swap(data);
    return true;
}

void cache_write(const std::string& path, const CacheKey& k, const std::vector<char>& cubin)
{
    // written under a name of its own, then renamed: readers see a whole file or none
    const std::string tmp = path + ".tmp" + std::to_string((long long)getpid()) + "_" +
                            std::to_string(std::hash<std::thread::id>()(std::this_thread::get_id()));
    {
        std::ofstream f(tmp, std::ios::binary | std::ios::trunc);
        if (!f) return;
        const uint64_t size = cubin.size(), sum = fnv1a(cubin.data(), cubin.size(), 0xCBF29CE484222325ull);
        f.write("FNJC", 4);
        f.write(reinterpret_cast<const char*>(&kCacheFormat), 4);
        f.write(reinterpret_cast<const char*>(&k.a), 8);
        f.write(reinterpret_cast<const char*>(&k.b), 8);
        f.write(reinterpret_cast<const char*>(&size), 8);
        f.write(cubin.data(), (std::streamsize)cubin.size());
        f.write(reinterpret_cast<const char*>(&sum), 8);
        if (!f) { f.close(); std::remove(tmp.c_str()); return; }
    }
    if (std::rename(tmp.c_str(), path.c_str()) != 0) std::remove(tmp.c_str());
}

// A module from the cache only (no compile); false on a miss.
bool cached_cubin(const ModuleSource& src, std::vector<char>& cubin)
{
    const std::string dir = cache_dir();
    if (dir.empty()) return false;
    const CacheKey k = cache_key(src);
    if (!cache_read(cache_path(dir, k), k, cubin)) return false;
    g_cache_hits.fetch_add(1);
    return true;
}

}  // namespace

void jit_cache_set_dir(const char* dir)
{
    std::lock_guard<std::mutex> lk(g_cache_mu);
    g_cache_resolved = true;
    g_cache_dir = (!dir || !*dir || std::strcmp(dir, "off") == 0) ? std::string() : std::string(dir);
    if (!g_cache_dir.empty()) make_dirs(g_cache_dir);
}

std::string jit_cache_dir() { return cache_dir(); }

void jit_cache_stats(unsigned long long* hits, unsigned long long* misses)
{
    if (hits) *hits = g_cache_hits.load();
    if (misses) *misses = g_cache_misses.load();
}

namespace {

// A compiled module: the number of programs, their sizes, their cubins, each from a multiple of 16 bytes.
size_t part_start(size_t pos) { return (pos + 15) / 16 * 16; }
std::vector<char> pack_parts(const std::vector<std::vector<char>>& parts)
{
    std::vector<uint64_t> head{(uint64_t)parts.size()};
    for (auto& p : parts) head.push_back(p.size());
    const char* h = reinterpret_cast<const char*>(head.data());
    std::vector<char> out(h, h + head.size() * sizeof(uint64_t));
    for (auto& p : parts) {
        out.resize(part_start(out.size()));
        out.insert(out.end(), p.begin(), p.end());
    }
    return out;
}

// Whether a compiled module is whole; `at` gets where each cubin begins.
bool unpack_parts(const std::vector<char>& module, std::vector<size_t>& at)
{
    at.clear();
    uint64_t n = 0, size = 0;
    if (module.size() < sizeof n) return false;
    std::memcpy(&n, module.data(), sizeof n);
    if (n == 0 || n > module.size() / sizeof n - 1) return false;
    size_t pos = (size_t)(n + 1) * sizeof n;
    for (uint64_t k = 0; k < n; ++k) {
        std::memcpy(&size, module.data() + (k + 1) * sizeof n, sizeof size);
        pos = part_start(pos);
        if (pos > module.size() || size > module.size() - pos) return false;
        at.push_back(pos);
        pos += (size_t)size;
    }
    return pos == module.size();
}

bool compile_program(const std::string& src, std::vector<char>& cubin, std::string& log)
{
    // FASTNOISE_JIT_VERBOSE=1 prints ptxas' register / spill report of every
    // specialised kernel to stderr (useful when tuning trees); it always compiles.
    const char* verbose = std::getenv("FASTNOISE_JIT_VERBOSE");
    const bool v = verbose && verbose[0] == '1';
    nvrtcProgram prog;
    if (nvrtcCreateProgram(&prog, src.c_str(), "fastnoise_jit.cu", 0, nullptr, nullptr) != NVRTC_SUCCESS) {
        log = "nvrtcCreateProgram failed";
        return false;
    }
    std::vector<const char*> opts(std::begin(kNvrtcOptions), std::end(kNvrtcOptions));
    if (v) opts.push_back("--ptxas-options=-v");
    nvrtcResult rc = nvrtcCompileProgram(prog, (int)opts.size(), opts.data());
    size_t loglen = 0;
    nvrtcGetProgramLogSize(prog, &loglen);
    log.assign(loglen, '\0');
    if (loglen) nvrtcGetProgramLog(prog, &log[0]);
    if (v) std::fprintf(stderr, "%s\n", log.c_str());
    if (rc != NVRTC_SUCCESS) {
        nvrtcDestroyProgram(&prog);
        return false;
    }
    size_t n = 0;
    nvrtcGetCUBINSize(prog, &n);
    cubin.resize(n);
    nvrtcGetCUBIN(prog, cubin.data());
    nvrtcDestroyProgram(&prog);
    return true;
}

}  // namespace

bool jit_compile_modules(const std::vector<ModuleSource>& modules, std::vector<std::vector<char>>& compiled, std::string& error)
{
    const char* verbose = std::getenv("FASTNOISE_JIT_VERBOSE");
    const bool v = verbose && verbose[0] == '1';
    compiled.assign(modules.size(), {});
    // NVRTC compiles independent programs concurrently, so they go to a pool of threads, the longest
    // first.  A program is a module's head with some of its parts: all of them, and the longest
    // programs in two until there is one for each thread (or a third more than modules), while they
    // take about as long as the head again (0.2 s, and 25 ms where the compiler has the program
    // cached).  FBm(Perlin) 3D takes 0.38 s (1.02 with one program per module, 0.62 without its column
    // kernels), the chunk mix's 16 programs 1.9 (4.3, 1.8; cached 0.79, 0.62, 0.47).
    unsigned nt = std::thread::hardware_concurrency();
    if (!nt) nt = 4;
    constexpr float kWorthSplitting = 0.15f;
    struct Unit {
        size_t module, first, end;               // its parts
        float seconds;
        std::vector<char> cubin;
    };
    std::vector<Unit> todo;
    auto estimate = [&](size_t m, size_t first, size_t end) {
        float t = 0;
        for (size_t k = first; k < end; ++k) t += modules[m].parts[k].seconds;
        return t;
    };
    for (size_t m = 0; m < modules.size(); ++m)
        todo.push_back(Unit{m, 0, modules[m].parts.size(), estimate(m, 0, modules[m].parts.size()), {}});
    const size_t most = std::max<size_t>(nt, todo.size() + todo.size() / 3 + 1);
    while (todo.size() < most) {
        Unit* longest = nullptr;
        for (Unit& u : todo)
            if (u.end - u.first > 1 && u.seconds > kWorthSplitting && (!longest || u.seconds > longest->seconds)) longest = &u;
        if (!longest) break;
        size_t at = longest->first + 1;          // as even as its parts allow, in their order
        while (at + 1 < longest->end && 2.0f * estimate(longest->module, longest->first, at) < longest->seconds) ++at;
        Unit rest{longest->module, at, longest->end, estimate(longest->module, at, longest->end), {}};
        longest->end = at;
        longest->seconds -= rest.seconds;
        todo.push_back(std::move(rest));
    }
    std::vector<char> cached(modules.size(), 0);
    for (size_t m = 0; !v && m < modules.size(); ++m) cached[m] = cached_cubin(modules[m], compiled[m]) ? 1 : 0;
    todo.erase(std::remove_if(todo.begin(), todo.end(), [&](const Unit& u) { return cached[u.module] != 0; }), todo.end());
    std::stable_sort(todo.begin(), todo.end(), [](const Unit& a, const Unit& b) { return a.seconds > b.seconds; });
    std::vector<std::string> logs(todo.size());
    std::vector<char> ok(todo.size(), 0);
    std::atomic<size_t> next{0};
    auto worker = [&]() {
        for (size_t i; (i = next.fetch_add(1)) < todo.size();) {
            const ModuleSource& m = modules[todo[i].module];
            std::string src = m.head;
            for (size_t k = todo[i].first; k < todo[i].end; ++k) src += m.parts[k].text;
            ok[i] = compile_program(src, todo[i].cubin, logs[i]) ? 1 : 0;
        }
    };
    nt = std::max(1u, std::min<unsigned>(nt, (unsigned)todo.size()));
    std::vector<std::thread> pool;
    for (unsigned t = 1; t < nt; ++t) pool.emplace_back(worker);
    worker();
    for (auto& t : pool) t.join();
    for (size_t i = 0; i < todo.size(); ++i)
        if (!ok[i]) { error = "NVRTC: " + logs[i].substr(0, 4000); return false; }
    const std::string dir = cache_dir();
    for (size_t m = 0; m < modules.size(); ++m) {
        std::vector<std::vector<char>> cubins;
        for (Unit& u : todo)
            if (u.module == m) cubins.push_back(std::move(u.cubin));
        if (cubins.empty()) continue;
        compiled[m] = pack_parts(cubins);
        g_cache_misses.fetch_add(1);
        if (!dir.empty()) {
            const CacheKey k = cache_key(modules[m]);
            cache_write(cache_path(dir, k), k, compiled[m]);
        }
    }
    return true;
}

bool jit_compile_all(const std::vector<const CompiledProgram*>& progs, std::vector<std::vector<char>>& compiled, std::string& error)
{
    std::vector<ModuleSource> modules{jit_batch_module(progs, 0)};
    for (auto* p : progs) modules.push_back(jit_percall_module(*p));
    return jit_compile_modules(modules, compiled, error);
}

namespace {

// A kernel of a module, whichever of its programs has it; false if none has.
bool find_kernel(const Module& m, const std::string& name, cudaKernel_t& out)
{
    for (cudaLibrary_t part : m.parts) {
        if (cudaLibraryGetKernel(&out, part, name.c_str()) == cudaSuccess) return true;
        cudaGetLastError();
    }
    return false;
}

// Load a compiled module.
std::unique_ptr<Module> load_module(const std::vector<char>& compiled, std::string& error)
{
    std::vector<size_t> at;
    if (!unpack_parts(compiled, at)) {
        error = "damaged module";
        return nullptr;
    }
    auto mod = std::make_unique<Module>();
    for (size_t pos : at) {
        cudaLibrary_t lib = nullptr;
        const cudaError_t e = cudaLibraryLoadData(&lib, compiled.data() + pos, nullptr, nullptr, 0, nullptr, nullptr, 0);
        if (e != cudaSuccess) {
            error = std::string("cudaLibraryLoadData: ") + cudaGetErrorString(e);
            return nullptr;
        }
        mod->parts.push_back(lib);
    }
    return mod;
}

// Load the batch module (compiled[0]) and the per-call modules (compiled[1 + k]) of `progs` and
// register their kernels.
bool jit_load(const std::vector<const CompiledProgram*>& progs, const std::vector<std::vector<char>>& compiled, std::string& error)
{
    std::vector<std::unique_ptr<Module>> mods;
    for (auto& c : compiled) {
        mods.push_back(load_module(c, error));
        if (!mods.back()) return false;
    }
    std::unordered_map<uint64_t, JitKernels> found;
    std::unordered_map<uint64_t, cudaKernel_t> batch;
    std::vector<ColPlan> plans;
    for (auto* p : progs) plans.push_back(column_plan(*p));
    bool ok = true;
    for (size_t k = 0; ok && k < progs.size(); ++k) {
        const Module& own = *mods[1 + k];
        JitKernels jk;
        jk.slot = (int)k;
        jk.column_step = plans[k].step;
        jk.point_cost = plans[k].point;
        for (auto& st : plans[k].states)
            jk.column_rates[jk.n_column_rates++] = st.rate;
        cudaKernel_t bk = nullptr;
        ok = find_kernel(own, "fnjit_grid_0", jk.grid) && find_kernel(own, "fnjit_pos_0", jk.positions) &&
             (progs[k]->dim != 4 || find_kernel(own, "fnjit_tile_0", jk.tileable)) &&
             (progs[k]->dim != 3 || (find_kernel(own, "fnjit_solid_0", jk.solid) && find_kernel(own, "fnjit_list_0", jk.list))) &&
             (plans[k].states.empty() || (find_kernel(own, "fnjit_col_0", jk.column) &&
                                          find_kernel(*mods[0], "fnjit_bcol_" + std::to_string(k), jk.batch_column))) &&
             find_kernel(*mods[0], "fnjit_batch_" + std::to_string(k), bk);
        const cudaKernel_t kern[4] = {jk.grid, jk.positions, jk.tileable, jk.column};
        for (int j = 0; ok && j < 4; ++j) {
            int n = 0;
            if (kern[j] && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, (const void*)kern[j], 256, 0) == cudaSuccess && n > 0)
                (j < 3 ? jk.resident[j] : jk.column_resident) = n;
            else
                cudaGetLastError();
        }
        found[progs[k]->hash] = jk;
        batch[progs[k]->hash] = bk;
    }
    if (!ok) {
        error = "kernel lookup failed in a specialised module";
        return false;
    }
    std::lock_guard<std::mutex> lk(g_jit_mu);
    for (auto& kv : found) g_kernels[kv.first] = kv.second;
    for (auto& kv : batch) {
        g_batch_kernels[kv.first] = kv.second;
        auto& vars = g_batch_variant_kernels[kv.first];
        vars.resize(batch_variants().size());
        vars[0] = BatchKernel{kv.second, batch_variants()[0].threads};
    }
    for (auto& m : mods) g_modules.push_back(std::move(m));   // modules stay loaded: kernels may still be queued
    return true;
}

std::mutex g_build_mu;                           // one build per program, even with concurrent first calls

}  // namespace

bool jit_build(const std::vector<const CompiledProgram*>& progs, std::string& error)
{
    if (progs.empty()) return true;
    std::vector<std::vector<char>> cubins;
    if (!jit_compile_all(progs, cubins, error)) return false;
    return jit_load(progs, cubins, error);
}

bool jit_try_cached(const CompiledProgram* prog)
{
    if (!prog || !g_enabled.load(std::memory_order_relaxed) || cache_dir().empty()) return false;
    static std::mutex tried_mu;
    static std::unordered_set<uint64_t> tried;          // one look per program and process
    {
        std::lock_guard<std::mutex> lk(tried_mu);
        if (!tried.insert(prog->hash).second) return false;
    }
    std::lock_guard<std::mutex> lk(g_build_mu);
    {
        std::lock_guard<std::mutex> rk(g_jit_mu);
        if (g_kernels.count(prog->hash) && g_batch_kernels.count(prog->hash)) return true;
    }
    std::vector<std::vector<char>> cubins(2);
    if (!cached_cubin(jit_batch_module({prog}, 0), cubins[0]) || !cached_cubin(jit_percall_module(*prog), cubins[1])) return false;
    std::string err;
    return jit_load({prog}, cubins, err);
}

bool jit_build_batch_variants(const std::vector<const CompiledProgram*>& progs, std::string& error)
{
    const size_t nv = batch_variants().size();
    std::vector<const CompiledProgram*> todo;
    {
        std::lock_guard<std::mutex> lk(g_jit_mu);
        for (auto* p : progs) {
            auto it = g_batch_variant_kernels.find(p->hash);
            bool all = it != g_batch_variant_kernels.end() && it->second.size() == nv;
            for (size_t v = 1; all && v < nv; ++v) all = it->second[v].kernel != nullptr;
            if (!all && std::find(todo.begin(), todo.end(), p) == todo.end()) todo.push_back(p);
        }
    }
    if (todo.empty()) return true;
    // one module per variant, compiled concurrently
    std::vector<ModuleSource> modules;
    for (size_t v = 1; v < nv; ++v) modules.push_back(jit_batch_module(todo, (int)v));
    std::vector<std::vector<char>> compiled;
    if (!jit_compile_modules(modules, compiled, error)) return false;
    std::vector<std::unique_ptr<Module>> mods;
    std::vector<std::vector<BatchKernel>> got(todo.size(), std::vector<BatchKernel>(nv));
    for (size_t i = 0; i < compiled.size(); ++i) {
        mods.push_back(load_module(compiled[i], error));
        if (!mods.back()) return false;
        const int v = (int)i + 1;
        for (size_t k = 0; k < todo.size(); ++k) {
            cudaKernel_t kern = nullptr;
            if (cudaLibraryGetKernel(&kern, mods.back()->parts[0], batch_kernel_name(k, v).c_str()) != cudaSuccess) {
                error = "kernel lookup failed in a batch variant module";
                return false;
            }
            got[k][(size_t)v] = BatchKernel{kern, batch_variants()[(size_t)v].threads};
        }
    }
    std::lock_guard<std::mutex> lk(g_jit_mu);
    for (size_t k = 0; k < todo.size(); ++k) {
        auto& vars = g_batch_variant_kernels[todo[k]->hash];
        vars.resize(nv);
        for (size_t v = 1; v < nv; ++v) vars[v] = got[k][v];
    }
    for (auto& m : mods) g_modules.push_back(std::move(m));
    return true;
}

bool jit_batch_kernel(uint64_t hash, int variant, BatchKernel& out)
{
    if (!g_enabled.load(std::memory_order_relaxed)) return false;
    std::lock_guard<std::mutex> lk(g_jit_mu);
    auto it = g_batch_variant_kernels.find(hash);
    if (it == g_batch_variant_kernels.end() || variant < 0 || (size_t)variant >= it->second.size() ||
        !it->second[(size_t)variant].kernel)
        return false;
    out = it->second[(size_t)variant];
    return true;
}

bool jit_lookup(uint64_t hash, JitKernels& out)
{
    if (!g_enabled.load(std::memory_order_relaxed)) return false;
    std::lock_guard<std::mutex> lk(g_jit_mu);
    auto it = g_kernels.find(hash);
    if (it == g_kernels.end()) return false;
    out = it->second;
    return true;
}

namespace {
bool is_built(uint64_t hash)
{
    std::lock_guard<std::mutex> lk(g_jit_mu);
    return g_kernels.count(hash) && g_batch_kernels.count(hash);
}
}  // namespace

bool jit_ensure(const CompiledProgram* prog, std::string& error)
{
    if (!prog->needs_specialisation()) return true;
    if (!g_enabled.load()) {
        error = "the tree evaluates a node per cell (node-driven Minkowski P), which only specialised kernels "
                "can do, and specialisation is disabled";
        return false;
    }
    std::lock_guard<std::mutex> lk(g_build_mu);
    {
        std::lock_guard<std::mutex> rk(g_jit_mu);
        if (g_kernels.count(prog->hash) && g_batch_kernels.count(prog->hash)) return true;
    }
    return jit_build({prog}, error);
}

void jit_set_enabled(bool on) { g_enabled.store(on); }
bool jit_enabled() { return g_enabled.load(); }

// ---------------------------------------------------------------- automatic specialisation
namespace {

struct AutoJit {
    std::mutex mu;
    std::condition_variable cv, idle_cv;
    std::unordered_map<uint64_t, int> uses;        // interpreter launches per program hash
    std::unordered_set<uint64_t> queued;           // handed to the worker once, whatever the outcome
    struct Job {
        CompiledProgram prog;                      // a copy: the caller's may go away
        int device;
        bool variants;                             // build the batch variants, not the tree's kernels
    };
    std::deque<Job> work;
    std::unordered_set<uint64_t> variants_queued;
    int running = 0;
    int threshold = -1;                            // -1 = not read from the environment yet
    bool stop = false;
    std::thread worker;
    ~AutoJit()
    {
        {
            std::lock_guard<std::mutex> lk(mu);
            stop = true;
            work.clear();
        }
        cv.notify_all();
        if (worker.joinable()) worker.join();
    }
};

AutoJit& auto_jit()
{
    static AutoJit a;
    return a;
}

int threshold_locked(AutoJit& a)
{
    if (a.threshold < 0) {
        const char* env = std::getenv("FASTNOISE_AUTO_SPECIALISE");
        a.threshold = env && *env ? std::max(0, std::atoi(env)) : 4;
    }
    return a.threshold;
}

void auto_worker()
{
    AutoJit& a = auto_jit();
    std::unique_lock<std::mutex> lk(a.mu);
    for (;;) {
        a.cv.wait(lk, [&] { return a.stop || !a.work.empty(); });
        if (a.stop) return;
        AutoJit::Job job = std::move(a.work.front());
        a.work.pop_front();
        ++a.running;
        lk.unlock();
        cudaSetDevice(job.device);
        std::string err;
        if (job.variants) {
            if (is_built(job.prog.hash)) jit_build_batch_variants({&job.prog}, err);   // a failure keeps variant 0
        } else if (!is_built(job.prog.hash)) {
            jit_build({&job.prog}, err);           // a failure leaves the interpreter in use
        }
        lk.lock();
        --a.running;
        if (a.work.empty() && a.running == 0) a.idle_cv.notify_all();
    }
}

}  // namespace

bool jit_is_specialised(uint64_t hash)
{
    std::lock_guard<std::mutex> lk(g_jit_mu);
    return g_kernels.count(hash) && g_batch_kernels.count(hash);
}

void jit_note_interpreted(const CompiledProgram* prog)
{
    if (!prog || !g_enabled.load(std::memory_order_relaxed)) return;
    AutoJit& a = auto_jit();
    std::lock_guard<std::mutex> lk(a.mu);
    const int t = threshold_locked(a);
    if (t == 0 || a.stop || a.queued.count(prog->hash)) return;
    if (++a.uses[prog->hash] < t) return;
    a.queued.insert(prog->hash);
    a.uses.erase(prog->hash);
    int dev = 0;
    cudaGetDevice(&dev);
    a.work.push_back(AutoJit::Job{*prog, dev, false});
    if (!a.worker.joinable()) a.worker = std::thread(auto_worker);
    a.cv.notify_one();
}

void jit_request_batch_variants(const CompiledProgram* prog)
{
    if (!prog || !g_enabled.load(std::memory_order_relaxed)) return;
    AutoJit& a = auto_jit();
    std::lock_guard<std::mutex> lk(a.mu);
    if (a.stop || a.variants_queued.count(prog->hash)) return;
    a.variants_queued.insert(prog->hash);
    int dev = 0;
    cudaGetDevice(&dev);
    a.work.push_back(AutoJit::Job{*prog, dev, true});
    if (!a.worker.joinable()) a.worker = std::thread(auto_worker);
    a.cv.notify_one();
}

int jit_set_auto_threshold(int uses)
{
    AutoJit& a = auto_jit();
    std::lock_guard<std::mutex> lk(a.mu);
    const int was = threshold_locked(a);
    a.threshold = std::max(0, uses);
    return was;
}

bool jit_auto_wait(int timeout_ms)
{
    AutoJit& a = auto_jit();
    std::unique_lock<std::mutex> lk(a.mu);
    auto idle = [&] { return a.work.empty() && a.running == 0; };
    if (timeout_ms < 0) {
        a.idle_cv.wait(lk, idle);
        return true;
    }
    return a.idle_cv.wait_for(lk, std::chrono::milliseconds(timeout_ms), idle);
}

GridRoute& grid_route()
{
    thread_local GridRoute r;
    return r;
}

namespace {

// The plane and steps of a grid.  A tree without a column kernel, other point sources and partial
// planes are not walked.
bool column_shape(const PointArgs& a, const JitKernels& jk, ColumnShape& shape)
{
    if (a.src != kSrcGrid || a.total <= 0 || a.total > (1ll << 31) || !jk.column) return false;
    long long plane = 1;
    for (int k = 0; k < a.dim - 1; ++k) plane *= a.count[k];
    if (plane <= 0) return false;
    const bool whole = !a.base && a.total == plane * a.count[a.dim - 1];
    if (!whole && (a.total % plane || a.base % plane)) return false;
    shape.plane = (unsigned)plane;
    shape.steps = whole ? (unsigned)a.count[a.dim - 1] : (unsigned)(a.total / plane);
    shape.first = a.base ? a.base / (unsigned)plane : 0u;
    return true;
}

// What a grid costs in columns, in issue slots.  A lattice state rebuilds a plane where a step enters
// the next cell, and both where it skips one.  A cellular or warp state builds one neighbourhood per
// distinct cell of a warp's lanes; where there are more than it has room for, the unit takes the
// state's point function.
void column_costs(const PointArgs& a, const JitKernels& jk, ColumnShape& shape)
{
    shape.step = jk.column_step;
    shape.enter = shape.cross = 0.0f;
    float slowest = jk.column_step;            // a step of a warp without room
    bool crowded = false;
    for (int k = 0; k < jk.n_column_rates; ++k) {
        const ColumnRate& c = jk.column_rates[k];
        const float r = std::fabs(c.scale[a.dim - 1] * a.step[a.dim - 1]), rate = r < 1.0f ? r : 1.0f;
        if (!c.cellular) {
            shape.enter += 2.0f * c.enter;
            shape.cross += c.enter * (r < 2.0f ? r : 2.0f);
            continue;
        }
        // the mean number of cells of a warp, the most, and the share of warps with more than four: of
        // 32 lanes in one row, of lanes at the end of a row and the beginning of the next, or of rows
        // shorter than a warp
        const float across = std::fabs(c.scale[0] * a.step[0]);
        const int n = a.count[0];
        auto share = [](float x) { return std::min(std::max(x, 0.0f), 1.0f); };
        const float span = (float)(std::min(n, 32) - 1) * across;
        float cells = 1.0f + span, most = 2.0f + std::floor(span), full = share(span - 3.0f);
        if (a.dim > 2 && n >= 32 && n % 32) {
            const float split = std::min(1.0f, 31.0f / (float)n);
            cells += split;
            most += 2.0f;
            full += split * (share(0.45f * (span - 0.8f)) - full);
        } else if (a.dim > 2 && n < 32) {
            cells *= 1.0f + (float)(31 / n + 1) * std::fabs(c.scale[1] * a.step[1]);
            most *= 2.0f;
            full = share(0.5f * (cells - 2.8f));
        }
        cells = std::min(cells, 4.0f);
        shape.enter += cells * c.enter;
        shape.cross += cells * c.enter * rate;
        // (with the few warps of these kernels, and neighbourhoods built in vain, a point costs more)
        shape.step += full * (2.5f * c.point - c.step);
        if (!(most <= 4.0f)) {
            slowest += c.point - c.step;
            crowded = true;
        }
    }
    // of one warp, beside others: a step's chain of loads and shuffles, and its issue
    shape.step_us = 0.006f + 0.008f * (float)jk.n_column_rates + shape.step / 980.0f + shape.cross / 800.0f;
    if (crowded) shape.step_us = std::max(shape.step_us, slowest / 400.0f);
}

// Issue slots of a unit of `len` steps, and what a microsecond issues: an SM, which the few warps
// of a kernel with one block per SM do not fill, times the SMs.
float column_unit_work(const ColumnShape& s, unsigned len) { return 250.0f + s.enter + (float)len * (s.step + s.cross); }
float slots_per_us() { return 9000.0f * (float)num_sms(); }
float column_slots_per_us(const JitKernels& jk) { return slots_per_us() / (jk.column_resident > 1 ? 1.0f : 1.3f); }

// Cut the columns into units of at most `len` steps, evenly.
void column_cut(ColumnShape& s, unsigned len)
{
    const unsigned segs = (s.steps + len - 1) / len;
    s.len = (s.steps + segs - 1) / segs;
    s.units = column_chunks(s) * ((s.steps + s.len - 1) / s.len);
}

// Cut a launch that has the GPU to itself, and say whether walking it in columns is faster than
// the point kernel.
//
// A launch takes what the units of the busiest SM issue, and the steps of a unit one after another;
// the two overlap in part (the root of the sum of their squares, over 1120 random grids within
// 16 %), and are the same where an SM has one block and no room for another.  Long units save
// entering cells (FBm(Perlin) 256^3 takes 221, 170, 147 us at 8, 16, 32 steps a unit), short ones
// spread over the SMs.
//
// Launches into device memory: about 3 us each more than that for a column kernel and 1.5, at least
// 3, for the point kernel, with which launches overlap better.  Back to back, point / column kernel,
// us: FBm(Perlin) 32^3 3.3 / 7.2, 96^3 19.9 / 14.0; CellularValue 64^3 9.0 / 6.6; terrain 64^3
// 21.5 / 26.7, 96^3 71 / 55; FBm(Value) of 5 octaves 1076 x 2092 at step 3.3 19.0 / 30.6.
//
// Host outputs: the caller waits for each, and large ones run at the host link, which a column's
// 128-byte rows use less well than the point kernel's runs of 512 bytes, above all where they do
// not start on a row of the link's (planes that are no multiple of 32) or in pageable memory (us of
// the call: CellularValue 32^3 15.1 / 14.2, Perlin 2D 2371 x 555 44 / 53, CellularValue 128^3 64 / 56;
// pageable Value 128^3 60 / 70, CellularDistance 90 / 74).
bool column_cut_alone(ColumnShape& s, const JitKernels& jk, OutputMemory memory)
{
    const unsigned n = s.steps, chunks = column_chunks(s), slots = 8u * (unsigned)num_sms();
    unsigned best = 1;
    float column_us = 1e30f;
    for (unsigned w = 1; w <= 16; ++w) {
        const unsigned fit = std::min(n, std::max(1u, w * slots / chunks)), len = (n + fit - 1) / fit;
        const unsigned long long units = (unsigned long long)chunks * ((n + len - 1) / len);
        const unsigned load = (unsigned)((units + slots - 1) / slots);
        const float issue = (float)load * (float)slots * column_unit_work(s, len) / column_slots_per_us(jk);
        const float chain = (float)len * s.step_us + s.enter / 3000.0f;
        const float us = load == 1 && jk.column_resident == 1 ? std::max(issue, chain) : std::sqrt(issue * issue + chain * chain);
        if (us < column_us) { column_us = us; best = len; }
        if (len == 1) break;
    }
    column_cut(s, best);
    const float points = (float)s.plane * (float)s.steps, bytes = 4.0f * points;
    const float point_us = points / 32.0f * jk.point_cost / slots_per_us();
    if (memory == kDeviceMemory) return column_us + 3.0f < 0.95f * std::max(point_us + 1.5f, 3.0f);
    column_us = std::max(column_us, bytes / (memory == kPageLocked && s.plane % 32u == 0 ? 190e3f : 130e3f));
    return column_us + 0.5f < 0.95f * std::max(std::max(point_us, jk.point_cost / 600.0f), bytes / 171e3f);
}

// Whether a launch of its own walks a grid in columns, and its shape if so.
bool column_alone(const PointArgs& a, const JitKernels& jk, OutputMemory memory, ColumnShape& s)
{
    const GridRoute& r = grid_route();
    if (r.route == FN_GRID_ROUTE_POINTS || !column_shape(a, jk, s)) return false;
    const bool asked = r.route == FN_GRID_ROUTE_COLUMNS;
    column_costs(a, jk, s);
    const bool faster = column_cut_alone(s, jk, memory);
    if (r.steps) column_cut(s, r.steps);
    return faster || asked;
}

}  // namespace

// A request's steps in units as column_tiles cuts them, against its points less a tenth for the
// estimates' errors.  A plane that is no multiple of 32 leaves lanes idle at every step.  Columns /
// points, us: 128 requests of FBm(Perlin) 2 x 50000 1409 / 228, 12 x 8000 287 / 219, 24 x 4000
// 167 / 219; of terrain 3 x 3 x 10000 2299 / 955, 33 x 3000 664 / 481; 64 of FBm(Perlin)
// 32 x 32 x 32 x 2 380 / 250, 1000 x 62 at 0.5 crossings 111 / 92.
bool jit_batch_columns(const PointArgs& a, const JitKernels& jk, ColumnShape& s, float& point_us, float& column_us)
{
    const GridRoute& r = grid_route();
    if (!jk.batch_column || r.route == FN_GRID_ROUTE_POINTS || !column_shape(a, jk, s)) return false;
    column_costs(a, jk, s);
    const unsigned chunks = column_chunks(s);
    unsigned len = s.steps < 16u ? s.steps : 16u;
    if ((unsigned long long)chunks * s.steps < 8ull * len) len = (chunks * s.steps + 7u) / 8u;
    column_us = (float)chunks * (float)((s.steps + len - 1) / len) * column_unit_work(s, len) / column_slots_per_us(jk);
    point_us = 0.9f * (float)s.plane * (float)s.steps / 32.0f * jk.point_cost / slots_per_us();
    return std::isfinite(point_us - column_us);   // infinite and NaN steps: points
}

unsigned column_tiles(ColumnShape& s, unsigned len)
{
    if (grid_route().steps) {
        column_cut(s, grid_route().steps);
        return (s.units + 7) / 8;
    }
    // a request with fewer units than a block has warps is cut finer
    const unsigned long long work = (unsigned long long)column_chunks(s) * s.steps;
    column_cut(s, (unsigned)std::max<unsigned long long>(1, std::min<unsigned long long>(len, (work + 7) / 8)));
    return (s.units + 7) / 8;
}

void column_args(PointArgs& a, const ColumnShape& s)
{
    a.col_plane = s.plane;
    a.col_steps = s.steps;
    a.col_first = s.first;
    a.col_len = s.len;
    a.col_units = s.units;
}

// Launch a per-call kernel so that it may start while the stream's previous kernel drains
// (programmatic dependent launch): its blocks take free SM slots, compute their first points
// and wait for that kernel before they touch memory (fne::wait_for_stream).
cudaError_t launch_overlapped(cudaKernel_t k, unsigned grid, void** params, cudaStream_t stream)
{
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(256);
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, (const void*)k, params);
}

// Whether the launch behind a column or position kernel of `blocks` may begin at once: where its
// blocks fill the SMs.  Where they leave SMs free, the next launch's blocks would take what is left of the
// occupied SMs too, run with them and crowd there, launch after launch; so it begins behind the
// points.  Back to back, us, at once / behind: terrain 2D 669 x 1365 in units of 32 steps (0.7
// blocks per SM) 104 / 52, of 16 (1.5) 62 / 35; CellularLookup 2D 1054 x 519 15.0 / 8.8; terrain 4D
// at 30000 positions 42 / 25; blend at 1 M positions (SMs full) 15.7 / 15.9.
unsigned begin_early(unsigned blocks, int resident) { return blocks >= (unsigned)(num_sms() * std::max(1, resident)) ? 1u : 0u; }

bool jit_launch(uint64_t hash, const PointArgs& args, float* out, MinMaxWork* work, float* dminmax, cudaStream_t stream,
                cudaError_t& err, OutputMemory memory)
{
    err = cudaSuccess;
    JitKernels jk;
    if (args.total <= 0 || args.total > (1ll << 31) || !jit_lookup(hash, jk)) return false;
    const int which = args.src == kSrcGrid ? 0 : args.src == kSrcPositions ? 1 : 2;
    ColumnShape shape;
    if (which == 0 && column_alone(args, jk, memory, shape)) {
        ++grid_route().columns;
        PointArgs c = args;
        column_args(c, shape);
        const unsigned grid = std::min<unsigned>((shape.units + 7) / 8, (unsigned)kMaxReduceBlocks);
        unsigned early = begin_early(grid, jk.column_resident);
        void* params[] = {&c, &out, &work, &dminmax, &early};
        err = launch_overlapped(jk.column, grid, params, stream);
        return true;
    }
    cudaKernel_t k = which == 0 ? jk.grid : which == 1 ? jk.positions : jk.tileable;
    if (!k) return false;
    const int sms = num_sms();
    unsigned ppl;
    long long blocks;
    if (args.total >= (long long)sms * 8 * 128 * 4) {
        // large calls: 4 points per lane (float4 stores), a grid of 8 blocks per SM striding over
        // the warp chunks
        ppl = 4u;
        blocks = std::min<long long>((args.total + 1023) / 1024, (long long)sms * 8);
    } else {
        // small calls are latency-bound: run them in one wave of the blocks that fit at once,
        // with as few points per lane as that allows (the fixed cost of a thread -- index set-up,
        // the min/max reduction -- is shared by its points)
        const long long resident = (long long)sms * std::max(1, jk.resident[which]) * 256;
        ppl = (unsigned)std::min<long long>(4, std::max<long long>(1, (args.total + resident - 1) / resident));
        blocks = (args.total + 256ll * ppl - 1) / (256ll * ppl);
    }
    if (blocks > kMaxReduceBlocks) blocks = kMaxReduceBlocks;
    if (blocks < 1) blocks = 1;
    PointArgs a = args;
    unsigned early = begin_early((unsigned)blocks, jk.resident[which]);
    void* params[] = {&a, &out, &work, &dminmax, &ppl, &early};
    err = launch_overlapped(k, (unsigned)blocks, params, stream);
    return true;
}

bool jit_launch_solid(uint64_t hash, const PointArgs& args, unsigned* above, unsigned* solid, MinMaxWork* work, float* dminmax,
                      float iso, cudaStream_t stream, cudaError_t& err)
{
    err = cudaSuccess;
    JitKernels jk;
    if (args.total <= 0 || args.total > (1ll << 31) || !jit_lookup(hash, jk) || !jk.solid) return false;
    const int sms = num_sms();
    unsigned ppl = 4u;                                     // the grid as the large per-call calls run it
    long long blocks = std::min<long long>((args.total + 1023) / 1024, (long long)sms * 8);
    if (args.total < (long long)sms * 8 * 128 * 4) {
        const long long resident = (long long)sms * std::max(1, jk.resident[0]) * 256;
        ppl = (unsigned)std::min<long long>(4, std::max<long long>(1, (args.total + resident - 1) / resident));
        blocks = (args.total + 256ll * ppl - 1) / (256ll * ppl);
    }
    if (blocks > kMaxReduceBlocks) blocks = kMaxReduceBlocks;
    if (blocks < 1) blocks = 1;
    PointArgs a = args;
    void* params[] = {&a, &above, &solid, &work, &dminmax, &iso, &ppl};
    err = cudaLaunchKernel((const void*)jk.solid, dim3((unsigned)blocks), dim3(256), params, 0, stream);
    return true;
}

bool jit_launch_list(uint64_t hash, const PointArgs& args, const unsigned* idx, const unsigned* count, unsigned max_count,
                     float* out, cudaStream_t stream, cudaError_t& err)
{
    err = cudaSuccess;
    JitKernels jk;
    if (args.total <= 0 || args.total > (1ll << 31) || !jit_lookup(hash, jk) || !jk.list) return false;
    long long blocks = std::min<long long>(((long long)max_count + 255) / 256, (long long)num_sms() * 8);
    if (blocks < 1) blocks = 1;
    PointArgs a = args;
    void* params[] = {&a, &idx, &count, &out};
    err = cudaLaunchKernel((const void*)jk.list, dim3((unsigned)blocks), dim3(256), params, 0, stream);
    return true;
}

}  // namespace fn
