// Shared by the sources of the library (not part of its interface).
#pragma once
#include <string>

namespace vesta_rt {
// records the text of a failure for vesta_last_error() and returns its code (never 0)
int fail(int code, const std::string& what);
// TMA descriptor of fp16 [d2][d1][d0] in boxes of box1 x 64 elements (d0 innermost), 128-byte swizzle, zeros outside
int tensor_map(void* out, const void* base, unsigned long long d0, unsigned long long d1, unsigned long long d2, unsigned box1);
// a pass bound for decode steps (pass.cu): `steps` steps on `stream`
int pass_steps(void* pass, void* stream, int steps);
}  // namespace vesta_rt
