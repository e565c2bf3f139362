// gsofa_fetch.h -- which device arrays share a copy on their way to the host.
#pragma once
#include <cstddef>

namespace gsofa {
namespace host {

// A device array and the caller's memory for it (null: not wanted).  `block`
// is the device allocation that the array is part of, null when it is one of
// its own.
struct Fetch {
    void* dst;
    const void* src;
    size_t bytes;
    const void* block;
};

constexpr int kMaxFetch = 8;
constexpr size_t kFetchStep = 256;  // arrays of one allocation start at multiples of this

// The copies into a staging buffer that bring all wanted arrays: array k lies
// at at[k] there.
struct FetchPlan {
    struct Copy {
        const char* src;
        size_t at, bytes;
    };
    Copy copy[kMaxFetch];
    int copies = 0;
    size_t at[kMaxFetch] = {};
    size_t bytes = 0;  // of the staging buffer
};

// One copy per run of arrays that lie one after another in the same
// allocation, with less than a step between them; what lies between belongs to
// that allocation too.  Arrays of different allocations never share a copy,
// however close they are: a copy must not run past the end of an allocation.
inline FetchPlan plan_fetch(const Fetch* f, int count) {
    FetchPlan p;
    const Fetch* prev = nullptr;
    for (int k = 0; k < count; k++) {
        if (!f[k].dst || !f[k].bytes) {
            prev = nullptr;
            continue;
        }
        const char* s = static_cast<const char*>(f[k].src);
        if (prev && prev->block && prev->block == f[k].block) {
            FetchPlan::Copy& c = p.copy[p.copies - 1];
            const char* end = c.src + c.bytes;
            if (s >= end && (size_t)(s - end) < kFetchStep) {
                p.at[k] = c.at + (size_t)(s - c.src);
                c.bytes = (size_t)(s - c.src) + f[k].bytes;
                p.bytes = c.at + c.bytes;
                prev = f + k;
                continue;
            }
        }
        p.at[k] = p.bytes;
        p.copy[p.copies++] = {s, p.bytes, f[k].bytes};
        p.bytes += f[k].bytes;
        prev = f + k;
    }
    return p;
}

}  // namespace host
}  // namespace gsofa
