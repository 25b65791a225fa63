// Whether an array in host memory is mapped to the GPU throughout.
#pragma once

#include <cstddef>
#include <cstdint>

namespace hf {

// one registration or allocation of host memory, [begin, end); begin == end: none
struct HostRange {
    uintptr_t begin, end;
};

// Whether ranges that kernels may address cover [p, p + bytes): range_at(q) gives the one that holds q.  (Both
// ends alone do not tell: an array may lie across two registrations with pages between them that are in none.)
template <class RangeAt>
bool host_covered(uintptr_t p, size_t bytes, RangeAt range_at) {
    const uintptr_t end = p + bytes;
    if (bytes == 0 || end < p) return false;
    while (p < end) {
        const HostRange r = range_at(p);
        if (p < r.begin || p >= r.end) return false;
        p = r.end;
    }
    return true;
}

}  // namespace hf
