// Two arrays that are of use only together: both, or neither.  Plain C++, so that
// the host can check it with an allocator that fails.
#pragma once
#include <cstddef>

// alloc(void **, bytes): 0 where it succeeds; release(void *)
template <class Alloc, class Release>
inline bool alloc_both(void **a, size_t a_bytes, void **b, size_t b_bytes, Alloc alloc, Release release) {
    *a = *b = nullptr;
    if (alloc(a, a_bytes) == 0) {
        if (alloc(b, b_bytes) == 0) return true;
        release(*a);
    }
    *a = *b = nullptr;
    return false;
}
