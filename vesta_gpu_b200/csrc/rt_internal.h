// Shared by the sources of the library (not part of its interface).
#pragma once
#include <string>

namespace vesta_rt {
// records the text of a failure for vesta_last_error() and returns its code (never 0)
int fail(int code, const std::string& what);
// TMA descriptor of fp16 [d2][d1][d0] (d0 innermost, the others `stride1` and `stride2` bytes apart) in boxes of
// box2 x box1 x 64 elements, 128-byte swizzle, zeros outside
int tensor_map(void* out, const void* base, unsigned long long d0, unsigned long long d1, unsigned long long d2,
               unsigned long long stride1, unsigned long long stride2, unsigned box1, unsigned box2);
// the same for rows [rows][fold] seen as [blocks of 64 fold indices][rows][64], in boxes of `blocks` blocks of `box_rows` rows
inline int fold_map(void* out, const void* base, unsigned long long fold, unsigned long long rows, unsigned box_rows, unsigned blocks) {
    return tensor_map(out, base, 64, rows, (fold + 63) / 64, fold * 2, 128, box_rows, blocks);
}
// a pass bound for decode steps (pass.cu): `steps` steps on `stream`
int pass_steps(void* pass, void* stream, int steps);
}  // namespace vesta_rt
