// Buffers that belong together, all or none.  No CUDA in here: the calls are the caller's, tests give their own.
#pragma once

#include <stddef.h>

namespace qkm {

struct Want {
    void** p;
    size_t bytes;
};

// Fills every *p by alloc(p, bytes), which returns 0 or an error.  On an error what was made is given back by release(*p), every *p is
// NULL again and the error is returned, so a later call starts anew.
template <int N, class Alloc, class Release>
inline int alloc_all(const Want (&want)[N], Alloc alloc, Release release) {
    for (int i = 0; i < N; ++i) {
        if (const int e = alloc(want[i].p, want[i].bytes)) {
            *want[i].p = nullptr;
            while (i-- > 0) {
                release(*want[i].p);
                *want[i].p = nullptr;
            }
            return e;
        }
    }
    return 0;
}

}  // namespace qkm
