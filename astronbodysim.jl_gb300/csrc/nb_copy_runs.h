// nb_copy_runs.h -- which of a download's host arrays go in one strided copy.
// Host code without CUDA calls, so that the choice can be checked on its own.
#pragma once

#include <stddef.h>
#include <stdint.h>

namespace nb {

// Addresses [lo, hi) of the pinned host allocation that holds an address; empty
// when there is none.
struct HostRange {
    uintptr_t lo = 0;
    uintptr_t hi = 0;
};

// Rows k, k + 1, ... that one strided copy may write, at least 1 (row k alone).
// dst, src: addresses of the rows (dst 0: not wanted), each of `bytes` bytes.
// The copy writes between its rows' ends as far as the driver knows, and knows
// one allocation only: the rows have to be evenly spaced at both ends, to
// follow each other without overlap, at most max_pitch apart, and to lie wholly
// in the pinned allocation of the first.  range_of(address) gives that, and is
// asked once, and only when there is more than one such row.
template <class RangeOf>
int copy_run(const uintptr_t* dst, const uintptr_t* src, int rows, int k, size_t bytes, size_t max_pitch,
             RangeOf range_of) {
    if (k + 1 >= rows || !dst[k] || !dst[k + 1] || dst[k + 1] <= dst[k] || src[k + 1] <= src[k]) return 1;
    const uintptr_t step = dst[k + 1] - dst[k], pitch = src[k + 1] - src[k];
    if (step < bytes || step > max_pitch || pitch < bytes || pitch > max_pitch) return 1;
    int run = 2;
    while (k + run < rows && dst[k + run] > dst[k + run - 1] && dst[k + run] - dst[k + run - 1] == step &&
           src[k + run] - src[k + run - 1] == pitch)
        ++run;
    const HostRange r = range_of(dst[k]);
    if (dst[k] < r.lo || dst[k] >= r.hi) return 1;
    while (run > 1 && r.hi - dst[k] < (uintptr_t)(run - 1) * step + bytes) --run;
    return run;
}

}  // namespace nb
