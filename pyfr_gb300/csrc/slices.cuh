// Memory that the slices of strided matrices take, for host code that decides
// which applies may run side by side.  Plain C++.
#pragma once

#include <stdint.h>

namespace b200 {

// n slices of rows x ld values, slice z at p + z stride (in values of 4 bytes)
struct Slices {
    const void *p;
    int64_t rows, ld, stride, n;
};

// Whether any slice of a and any slice of b, whole rows taken, share a value.
// With equal positive strides (several matrices' rows interleaved slice by
// slice) exactly; with others, whether the ranges from the first to the last
// slice do.
inline bool overlap(const Slices &a, const Slices &b) {
    const int64_t d = ((int64_t)(uintptr_t)b.p - (int64_t)(uintptr_t)a.p) / 4;
    const int64_t la = a.rows * a.ld, lb = b.rows * b.ld;
    if (!a.p || !b.p || la <= 0 || lb <= 0 || a.n <= 0 || b.n <= 0) return false;
    if (a.stride != b.stride || a.stride <= 0 || a.n == 1 || b.n == 1) {
        const int64_t ea = (a.n - 1) * a.stride, eb = (b.n - 1) * b.stride;
        const int64_t a0 = ea < 0 ? ea : 0, a1 = (ea < 0 ? 0 : ea) + la;
        const int64_t b0 = d + (eb < 0 ? eb : 0), b1 = d + (eb < 0 ? 0 : eb) + lb;
        return a0 < b1 && b0 < a1;
    }
    // Slice i of a and slice j of b are k = i - j strides apart: the first k whose
    // a-slice ends behind b's start decides
    const int64_t s = a.stride, x = d - la;
    int64_t k = (x >= 0 ? x / s : -((-x + s - 1) / s)) + 1;
    if (k < 1 - b.n) k = 1 - b.n;
    return k <= a.n - 1 && k * s < d + lb && d < k * s + la;
}

}  // namespace b200
