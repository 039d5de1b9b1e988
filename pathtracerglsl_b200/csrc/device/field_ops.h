// field_ops.h — the typed form of a coefficient field's program (host/field_compile.cpp writes
// it at upload, field_eval in occupants.cuh runs it).
//
// The C ABI's programs are stack programs of three-float values.  Most values are scalars that
// fill all three, so the typed form marks every operand as scalar or vector and computes a
// scalar once; it also multiplies and adds constants in place.  Every value is the one the
// untyped program computes.
#pragma once

namespace ptx {

enum FieldOp : unsigned {
    kFieldEnd, kFieldPushP, kFieldPushPV, kFieldPushC, kFieldPushCV, kFieldSwz, kFieldMulC, kFieldAddC,
    kFieldNeg, kFieldExp, kFieldLog, kFieldSin, kFieldCos, kFieldSqrt, kFieldAbs, kFieldFloor, kFieldFract, kFieldLength,
    kFieldAdd, kFieldSub, kFieldMul, kFieldDiv, kFieldPow, kFieldMin, kFieldMax, kFieldMod, kFieldStep, kFieldDot,
    kFieldClamp, kFieldMix, kFieldSmoothstep, kFieldVec3
};
// Word: the op in bits 0-7, flags, a component index in bits 16-17.  The operand nearest the
// stack's bottom is A, the top is the last one.
constexpr unsigned kFieldVec = 1u << 8;     // the result is a vector (the last result, for kFieldEnd)
constexpr unsigned kFieldA = 1u << 9;       // operand A is a vector (push: the value it covers is)
constexpr unsigned kFieldB = 1u << 10;      // operand B (binary: the top)
constexpr unsigned kFieldC = 1u << 11;      // operand C (ternary: the top)
constexpr unsigned kFieldSwap = 1u << 12;   // binary: A is the top
constexpr unsigned kFieldFirst = 1u << 13;  // push onto an empty stack

}  // namespace ptx
