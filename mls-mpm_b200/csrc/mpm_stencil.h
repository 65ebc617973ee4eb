// mpm_stencil.h — index tests of a 3x3x3 stencil around a cell.
//
// cell_frac saturates: a coordinate of 2^31 or more, or an infinity, gives the
// cell INT32_MAX (or INT32_MIN), next to which signed sums overflow and a test
// such as `c + 1 < n` answers true.  All arithmetic here is on u32, where it
// wraps by definition, so the answers hold for every cell.  Plain C++ outside
// nvcc.
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define MPM_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define MPM_HOST_DEVICE inline
#endif

namespace mpm {

// True when the cells c - 1, c and c + 1 of an axis lie in [lo, lo + n);
// 3 <= n and -1 <= lo, lo + n < 2^30.
MPM_HOST_DEVICE bool stencil_in(int32_t c, int32_t lo, int32_t n) {
    return (uint32_t)c - 1u - (uint32_t)lo < (uint32_t)n - 2u;
}

// Cell k = 0, 1, 2 of the stencil around c (c - 1 + k, wrapping: beyond
// INT32_MAX it is negative, below INT32_MIN beyond every grid).
MPM_HOST_DEVICE int32_t stencil_cell(int32_t c, int k) { return (int32_t)((uint32_t)c - 1u + (uint32_t)k); }

}  // namespace mpm
