"""Typed field programs (host/field_compile.cpp) compute the values of the stack programs they are
made from, bit for bit: the compiler and the device's interpreter (occupants.cuh field_eval) built
for the host beside an interpreter of the untyped program, over the expressions of the GPU test and
random programs of every operation, constant, operand form and depth."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from pathtracerglsl_b200 import field
from test_gpu_field_programs import SOURCES

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "pathtracerglsl_b200", "csrc")

HARNESS = r"""
#include <cmath>
#include <cstring>
#include "ptx_rt.h"
#include "device/field_ops.h"
#include "host/field_compile.h"
#define __device__
#define __noinline__
#define __forceinline__ inline
namespace ptx {
struct f3 {
    float x, y, z;
    f3() {}
    explicit f3(float v) : x(v), y(v), z(v) {}
    f3(float a, float b, float c) : x(a), y(b), z(c) {}
};
static float dot(f3 a, f3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
static unsigned __ldg(const uint32_t* p) { return *p; }
static float __uint_as_float(unsigned u) { float f; std::memcpy(&f, &u, 4); return f; }
static float m_exp(float x) { return std::exp(x); }
static float m_log(float x) { return std::log(x); }
static float m_sin(float x) { return std::sin(x); }
static float m_cos(float x) { return std::cos(x); }
static float m_pow(float x, float y) { return std::pow(x, y); }
@SOURCE@

// The untyped program: a stack of three floats per value.
static float one(uint32_t op, float x, float y, float z) {
    switch (op) {
        case PTR_FOP_ADD: return x + y;
        case PTR_FOP_SUB: return x - y;
        case PTR_FOP_MUL: return x * y;
        case PTR_FOP_DIV: return x / y;
        case PTR_FOP_NEG: return -x;
        case PTR_FOP_EXP: return m_exp(x);
        case PTR_FOP_LOG: return m_log(x);
        case PTR_FOP_SIN: return m_sin(x);
        case PTR_FOP_COS: return m_cos(x);
        case PTR_FOP_SQRT: return sqrtf(x);
        case PTR_FOP_ABS: return fabsf(x);
        case PTR_FOP_FLOOR: return floorf(x);
        case PTR_FOP_FRACT: return x - floorf(x);
        case PTR_FOP_POW: return m_pow(x, y);
        case PTR_FOP_MIN: return y < x ? y : x;
        case PTR_FOP_MAX: return x < y ? y : x;
        case PTR_FOP_MOD: return x - y * floorf(x / y);
        case PTR_FOP_STEP: return y < x ? 0.0f : 1.0f;
        case PTR_FOP_CLAMP: x = x < y ? y : x; return z < x ? z : x;
        case PTR_FOP_MIX: return x * (1.0f - z) + y * z;
        default: {   // smoothstep
            float t = (z - x) / (y - x);
            t = t < 0.0f ? 0.0f : (t > 1.0f ? 1.0f : t);
            return t * t * (3.0f - 2.0f * t);
        }
    }
}
static f3 untyped(const uint32_t* code, f3 p) {
    f3 st[PTR_FIELD_MAX_STACK];
    int sp = 0;
    for (;;) {
        const uint32_t op = *code++;
        if (op == PTR_FOP_END) return st[0];
        if (op == PTR_FOP_P) { st[sp++] = p; continue; }
        if (op == PTR_FOP_CONST) {
            st[sp++] = f3(__uint_as_float(code[0]), __uint_as_float(code[1]), __uint_as_float(code[2]));
            code += 3;
            continue;
        }
        f3& a = st[sp - 1];
        if (op == PTR_FOP_SWZ) {
            const uint32_t c = *code++;
            a = f3(c == 0 ? a.x : c == 1 ? a.y : a.z);
        } else if (op == PTR_FOP_LENGTH) {
            a = f3(sqrtf(dot(a, a)));
        } else if (op >= PTR_FOP_NEG && op <= PTR_FOP_FRACT) {
            a = f3(one(op, a.x, 0, 0), one(op, a.y, 0, 0), one(op, a.z, 0, 0));
        } else if (op == PTR_FOP_CLAMP || op == PTR_FOP_MIX || op == PTR_FOP_SMOOTHSTEP || op == PTR_FOP_VEC3) {
            const f3 z = st[--sp], y = st[--sp], x = st[sp - 1];
            st[sp - 1] = op == PTR_FOP_VEC3 ? f3(x.x, y.x, z.x) : f3(one(op, x.x, y.x, z.x), one(op, x.y, y.y, z.y), one(op, x.z, y.z, z.z));
        } else {
            const f3 y = st[--sp], x = st[sp - 1];
            st[sp - 1] = op == PTR_FOP_DOT ? f3(dot(x, y)) : f3(one(op, x.x, y.x, 0), one(op, x.y, y.y, 0), one(op, x.z, y.z, 0));
        }
    }
}
}  // namespace ptx
// Values of a program that starts at `start` at n points, untyped and typed.
extern "C" void evaluate(const uint32_t* code, int start, const float* p, int n, float* a, float* b) {
    const std::vector<uint32_t> typed = ptx_host::compile_field(code, start);
    for (int k = 0; k < n; ++k) {
        const ptx::f3 q(p[3 * k], p[3 * k + 1], p[3 * k + 2]);
        const ptx::f3 u = ptx::untyped(code + start, q), t = ptx::field_eval(typed.data(), q);
        a[3 * k] = u.x; a[3 * k + 1] = u.y; a[3 * k + 2] = u.z;
        b[3 * k] = t.x; b[3 * k + 1] = t.y; b[3 * k + 2] = t.z;
    }
}
"""


@pytest.fixture(scope="module")
def evaluate(tmp_path_factory):
    src = open(os.path.join(CSRC, "device", "occupants.cuh")).read()
    body = src[src.index("__device__ __forceinline__ float fract_"):src.index("__device__ __forceinline__ bool mat_is_het")]
    d = tmp_path_factory.mktemp("field")
    (d / "field.cpp").write_text(HARNESS.replace("@SOURCE@", body))
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-Wno-unknown-pragmas", "-shared", "-fPIC", "-I", CSRC,
                    "-I", os.path.join(ROOT, "include"), str(d / "field.cpp"), os.path.join(CSRC, "host", "field_compile.cpp"),
                    "-o", str(d / "field.so")], check=True)
    lib = C.CDLL(str(d / "field.so"))

    def run(code, points, start=0):
        code = np.ascontiguousarray(code, np.uint32)
        out = [np.zeros_like(points) for _ in range(2)]
        lib.evaluate(code.ctypes.data_as(C.c_void_p), start, points.ctypes.data_as(C.c_void_p), len(points),
                     *(o.ctypes.data_as(C.c_void_p) for o in out))
        return out
    return run


def _same(a, b):
    nan = np.isnan(a)
    np.testing.assert_array_equal(nan, np.isnan(b))
    np.testing.assert_array_equal(a.view(np.uint32)[~nan], b.view(np.uint32)[~nan])   # signed zeros too


def _points(rng, n):
    p = rng.uniform(-2.0, 2.0, (n, 3)).astype(np.float32)
    p[::7] *= 1e4
    p[::5] = np.round(p[::5])
    return p


@pytest.mark.parametrize("src", SOURCES)
def test_expressions(evaluate, src):
    code = field.compile_field({"kind": "glsl", "source": src}, {})
    _same(*evaluate(code, _points(np.random.RandomState(1), 300)))


END, CONST, P, SWZ = 0, 1, 2, 3
UNARY = list(range(8, 17)) + [26]            # NEG .. FRACT, LENGTH
BINARY = list(range(4, 8)) + list(range(17, 22)) + [25]
TERNARY = [22, 23, 24, 27]
VALUES = [0.0, -0.0, 1.0, -1.0, 0.5, 2.0, 0.3, 7.25, 1e-3, 1e30, 1e-42]


def _random_program(rng, depth):
    """A valid program: pushes, and operations the stack can serve, to one value."""
    bits = lambda v: int(np.float32(v).view(np.uint32))   # noqa: E731
    code, sp = [], 0
    for _ in range(int(rng.randint(1, 40))):
        ops = []
        if sp < depth:
            ops += ["push"] * 3
        if sp >= 1:
            ops += ["unary", "swz"]
        if sp >= 2:
            ops += ["binary"] * 3
        if sp >= 3:
            ops += ["ternary"] * 2
        op = ops[rng.randint(len(ops))]
        if op == "push":
            form = rng.randint(5)
            if form < 2:
                code += [CONST] + [bits(VALUES[rng.randint(len(VALUES))])] * 3
            elif form == 2:
                code += [CONST] + [bits(VALUES[rng.randint(len(VALUES))]) for _ in range(3)]
            elif form == 3:
                code += [P]
            else:
                code += [P, SWZ, int(rng.randint(3))]
            sp += 1
        elif op == "swz":
            code += [SWZ, int(rng.randint(3))]
        elif op == "unary":
            code.append(UNARY[rng.randint(len(UNARY))])
        elif op == "binary":
            code.append(BINARY[rng.randint(len(BINARY))])
            sp -= 1
        else:
            code.append(TERNARY[rng.randint(len(TERNARY))])
            sp -= 2
    while sp > 1:
        code.append(BINARY[rng.randint(len(BINARY))])
        sp -= 1
    return code + [END]


@pytest.mark.parametrize("depth", [1, 2, 3, 5, 16])
def test_random_programs(evaluate, depth):
    rng = np.random.RandomState(depth)
    points = _points(rng, 24)
    with np.errstate(all="ignore"):
        for _ in range(3000):
            head = [END] * int(rng.randint(3))   # programs lie anywhere in the table
            _same(*evaluate(head + _random_program(rng, depth), points, len(head)))
