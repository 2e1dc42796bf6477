// The order in which the small-d sweep starts its row tiles: a total order, so
// that the ranks of any set of extents are a permutation. (Plain C++: the host
// can check the rule.)
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define CG_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define CG_HOST_DEVICE inline
#endif

namespace culof_gb300 {

// Ordered key of an extent's float bits (a sum of squares: not negative, but
// inf - inf makes it not a number, which compares with nothing): what is not a
// number counts as the widest.
CG_HOST_DEVICE uint32_t extent_key(uint32_t float_bits) {
    const uint32_t u = float_bits & 0x7FFFFFFFu;
    return u > 0x7F800000u ? 0xFFFFFFFFu : u;
}

// Whether tile a starts before tile b: wider first, equal ones by number.
CG_HOST_DEVICE bool starts_before(uint32_t key_a, int a, uint32_t key_b, int b) {
    return key_a > key_b || (key_a == key_b && a < b);
}

}  // namespace culof_gb300
