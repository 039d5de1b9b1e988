// field_compile.h — typed coefficient-field programs (device/field_ops.h).
#pragma once
#include <cstdint>
#include <vector>

namespace ptx_host {

// The typed form of the validated stack program at code[start].
std::vector<uint32_t> compile_field(const uint32_t* code, int start);

}  // namespace ptx_host
