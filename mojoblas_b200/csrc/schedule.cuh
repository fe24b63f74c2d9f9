// Arithmetic of the kernels' schedules, for the host and the device: plain C++ with no CUDA in
// it, so that a host compiler can check it at sizes that no test can run
// (tests/test_schedule.py).
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define MBG_HD __host__ __device__ __forceinline__
#else
#define MBG_HD inline
#endif

typedef int64_t i64;

namespace mbg {

// A reduction of k elements in slabs of `depth`: n slabs, the last of `last` elements.  A kernel
// asks for what is left from a slab's start on, never for the start itself, which passes
// 2^31 in the last slab of a reduction near 2^31.
struct KSlabs {
    i64 n;
    int last;
};
MBG_HD KSlabs k_slabs(i64 k, int depth) {
    KSlabs s;
    s.n = (k + depth - 1) / depth;
    s.last = s.n ? int(k - (s.n - 1) * depth) : 0;
    return s;
}
MBG_HD int k_left(int nkb, int last, int kb, int depth) { return kb + 1 < nkb ? depth : last; }

}  // namespace mbg
