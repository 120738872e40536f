// Division by a run-time constant as one high product (no includes: the CPU tests
// compile this file as plain C++).
#pragma once

namespace cdns {

// x / d for 0 <= x, x d < 2^32, d >= 1: the high word of x ceil(2^32 / d).  The divisor
// 1 (a mesh without streamwise modes has one line of x) stands apart: its 2^32 does not
// fit the word.
struct FastDiv {
    unsigned m;
    int n;
    __host__ __device__ __forceinline__ explicit FastDiv(int d) : m(0xffffffffu / (unsigned)d + 1u), n(d) {}
    __host__ __device__ __forceinline__ int operator()(int x) const {
        if (n == 1) return x;
#ifdef __CUDA_ARCH__
        return (int)__umulhi((unsigned)x, m);
#else
        return (int)(((unsigned long long)(unsigned)x * m) >> 32);
#endif
    }
};

}  // namespace cdns
