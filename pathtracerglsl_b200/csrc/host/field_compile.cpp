// field_compile.cpp — a coefficient field's stack program (ptr_scene_desc.field_code) in its
// typed form: scalar values computed once, constants multiplied and added in place.
//
// Scalar constants stay off the machine's stack until an operation needs them there: a
// product or sum takes them as an immediate (both commute exactly), constant arithmetic folds
// in binary32 (+, -, *, / and negation round alike here and on the device), any other
// operation pushes them, with its operands swapped where the constant came first.  A
// three-operand operation whose constants lie below computed values recompiles with every
// constant pushed in place.
#include "field_compile.h"
#include <cstring>
#include "../device/field_ops.h"
#include "ptx_rt.h"

using namespace ptx;

namespace ptx_host {
namespace {

struct Value {
    bool vec;
    bool pending;   // a scalar constant not yet on the machine's stack
    float c;
};

float as_float(uint32_t w) { float f; std::memcpy(&f, &w, 4); return f; }
uint32_t as_word(float f) { uint32_t w; std::memcpy(&w, &f, 4); return w; }

struct Compiler {
    std::vector<uint32_t> out;
    std::vector<Value> st;
    bool lazy = true;

    // the machine's top, if any, below which a push goes
    uint32_t push_flags() const {
        for (size_t k = st.size(); k-- > 0;)
            if (!st[k].pending) return st[k].vec ? kFieldA : 0u;
        return kFieldFirst;
    }
    void push_const(float c) { out.push_back(kFieldPushC | push_flags()); out.push_back(as_word(c)); }
    // puts the top on the machine's stack
    void settle_top() {
        if (!st.back().pending) return;
        const float c = st.back().c;
        st.pop_back();
        push_const(c);
        st.push_back({false, false, 0.0f});
    }
    void immediate(unsigned op, const Value& v, float c) {
        out.push_back(op | (v.vec ? kFieldVec : 0u));
        out.push_back(as_word(c));
    }
    void binary(unsigned op) {
        const Value b = st.back(); st.pop_back();
        const Value a = st.back(); st.pop_back();
        const bool result_vec = op != kFieldDot && (a.vec || b.vec);
        if (a.pending && b.pending) {
            if (op == kFieldAdd || op == kFieldSub || op == kFieldMul || op == kFieldDiv) {
                const float c = op == kFieldAdd ? a.c + b.c : op == kFieldSub ? a.c - b.c : op == kFieldMul ? a.c * b.c : a.c / b.c;
                st.push_back({false, true, c});
                return;
            }
            push_const(a.c);
            st.push_back({false, false, 0.0f});
            push_const(b.c);
            st.pop_back();
        } else if ((op == kFieldMul || op == kFieldAdd) && (a.pending || b.pending)) {
            const Value& v = a.pending ? b : a;
            immediate(op == kFieldMul ? kFieldMulC : kFieldAddC, v, a.pending ? a.c : b.c);
            st.push_back({v.vec, false, 0.0f});
            return;
        } else if (b.pending) {
            st.push_back(a);
            push_const(b.c);
            st.pop_back();
        } else if (a.pending) {   // the machine's order is (b, a)
            st.push_back(b);
            push_const(a.c);
            st.pop_back();
            out.push_back(op | kFieldSwap | (result_vec ? kFieldVec : 0u) | (b.vec ? kFieldB : 0u));
            st.push_back({result_vec, false, 0.0f});
            return;
        }
        out.push_back(op | (result_vec ? kFieldVec : 0u) | (a.vec ? kFieldA : 0u) | (b.vec ? kFieldB : 0u));
        st.push_back({result_vec, false, 0.0f});
    }
    // false: a constant lies below a computed operand
    bool ternary(unsigned op) {
        Value v[3];
        for (int k = 2; k >= 0; --k) { v[k] = st.back(); st.pop_back(); }
        for (int k = 0; k < 3; ++k) {
            if (v[k].pending) push_const(v[k].c);
            else if (k > 0 && v[k - 1].pending) return false;
            st.push_back({v[k].vec, false, 0.0f});
        }
        for (int k = 0; k < 3; ++k) st.pop_back();
        const bool vec = op == kFieldVec3 || v[0].vec || v[1].vec || v[2].vec;
        out.push_back(op | (vec ? kFieldVec : 0u) | (v[0].vec ? kFieldA : 0u) | (v[1].vec ? kFieldB : 0u) | (v[2].vec ? kFieldC : 0u));
        st.push_back({vec, false, 0.0f});
        return true;
    }
    bool run(const uint32_t* code, int pc) {
        for (;;) {
            const uint32_t op = code[pc++];
            switch (op) {
                case PTR_FOP_END:
                    settle_top();
                    out.push_back(kFieldEnd | (st.back().vec ? kFieldVec : 0u));
                    return true;
                case PTR_FOP_CONST: {
                    const uint32_t x = code[pc], y = code[pc + 1], z = code[pc + 2];
                    pc += 3;
                    if (x == y && x == z) {
                        if (lazy) { st.push_back({false, true, as_float(x)}); break; }
                        push_const(as_float(x));
                        st.push_back({false, false, 0.0f});
                    } else {
                        out.push_back(kFieldPushCV | push_flags());
                        out.insert(out.end(), {x, y, z});
                        st.push_back({true, false, 0.0f});
                    }
                    break;
                }
                case PTR_FOP_P:
                    if (code[pc] == PTR_FOP_SWZ) {
                        out.push_back(kFieldPushP | push_flags() | (code[pc + 1] << 16));
                        pc += 2;
                        st.push_back({false, false, 0.0f});
                    } else {
                        out.push_back(kFieldPushPV | push_flags());
                        st.push_back({true, false, 0.0f});
                    }
                    break;
                case PTR_FOP_SWZ: {
                    const uint32_t c = code[pc++];
                    if (!st.back().vec) break;   // every component of a scalar is the scalar
                    out.push_back(kFieldSwz | (c << 16));
                    st.back().vec = false;
                    break;
                }
                case PTR_FOP_NEG:
                    if (st.back().pending) { st.back().c = -st.back().c; break; }
                    out.push_back(kFieldNeg | (st.back().vec ? kFieldVec : 0u));
                    break;
                case PTR_FOP_EXP: case PTR_FOP_LOG: case PTR_FOP_SIN: case PTR_FOP_COS: case PTR_FOP_SQRT: case PTR_FOP_ABS:
                case PTR_FOP_FLOOR: case PTR_FOP_FRACT:
                    settle_top();
                    out.push_back((kFieldExp + (op - PTR_FOP_EXP)) | (st.back().vec ? kFieldVec : 0u));
                    break;
                case PTR_FOP_LENGTH:
                    settle_top();
                    out.push_back(kFieldLength | (st.back().vec ? kFieldA : 0u));
                    st.back().vec = false;
                    break;
                case PTR_FOP_ADD: binary(kFieldAdd); break;
                case PTR_FOP_SUB: binary(kFieldSub); break;
                case PTR_FOP_MUL: binary(kFieldMul); break;
                case PTR_FOP_DIV: binary(kFieldDiv); break;
                case PTR_FOP_POW: binary(kFieldPow); break;
                case PTR_FOP_MIN: binary(kFieldMin); break;
                case PTR_FOP_MAX: binary(kFieldMax); break;
                case PTR_FOP_MOD: binary(kFieldMod); break;
                case PTR_FOP_STEP: binary(kFieldStep); break;
                case PTR_FOP_DOT: binary(kFieldDot); break;
                case PTR_FOP_CLAMP: if (!ternary(kFieldClamp)) return false; break;
                case PTR_FOP_MIX: if (!ternary(kFieldMix)) return false; break;
                case PTR_FOP_SMOOTHSTEP: if (!ternary(kFieldSmoothstep)) return false; break;
                default: if (!ternary(kFieldVec3)) return false; break;   // PTR_FOP_VEC3
            }
        }
    }
};

}  // namespace

std::vector<uint32_t> compile_field(const uint32_t* code, int start) {
    Compiler c;
    if (!c.run(code, start)) {
        c = Compiler();
        c.lazy = false;
        c.run(code, start);
    }
    return c.out;
}

}  // namespace ptx_host
