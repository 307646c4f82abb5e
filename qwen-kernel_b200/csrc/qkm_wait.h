// A thread's record of its bounded waits.  Compiles for the host too, where tests walk it.
#pragma once

#ifdef __CUDACC__
#define QKM_HD __host__ __device__ __forceinline__
#else
#define QKM_HD inline
#endif

namespace qkm {

struct Waits {
    bool out = false;   // a wait has run out; stays set

    // w(): waits, false if it ran out.  Once one has, no other is waited for: a thread spends the limit once.
    template <class W>
    QKM_HD void wait(W w) {
        if (!(out || w())) out = true;   // (written `if (!out) out = !w()` it cost the GEMM kernel 16 bytes of spills and 1 %)
    }
    // Before the next unit of a work list is taken: false when a wait has run out, this one or an earlier one, in any thread that
    // any() asks; the unit must not be read then.
    template <class W, class Any>
    QKM_HD bool next(W w, Any any) {
        wait(w);
        out = any(out);
        return !out;
    }
};

}  // namespace qkm
