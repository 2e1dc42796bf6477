// Per-row candidate lists held by one warp, and a finished row's output.
#pragma once

#include <stdint.h>

#include "common.cuh"
#include "warp_sort.cuh"

namespace culof_gb300 {

constexpr unsigned kFullMask = 0xffffffffu;
constexpr int kInsertMax = 12;  // more new keys than this are sorted and merged

__device__ __forceinline__ float inf_f() { return __int_as_float(0x7f800000); }

// A row's list: its 32 * KR best keys so far in ascending order, element
// e = 32 j + lane in register b[j] while a warp works on it.

// Merges up to 32 keys, one per lane (kKeyMax: none), into the list (about 250
// issue slots).
template <int KR>
__device__ __forceinline__ void list_merge(uint64_t (&b)[KR], uint64_t key) {
    const int lane = threadIdx.x & 31;
    uint64_t x[1] = {key};
    warp_bitonic_sort<1>(x);
    if constexpr (KR == 1) {
        b[0] = warp_merge_lowest32(b[0], x[0]);
    } else {
        // the 32 best of (second register, new keys), then both runs of 32
        // merged into 64: elementwise minimum and maximum against the
        // reversed run, each a bitonic sequence
        const uint64_t c = warp_merge_lowest32(b[1], x[0]);
        const uint64_t rc = __shfl_sync(kFullMask, c, 31 - lane);
        uint64_t lo = b[0] < rc ? b[0] : rc, hi = b[0] < rc ? rc : b[0];
#pragma unroll
        for (int st = 16; st > 0; st >>= 1) {
            const uint64_t ol = shfl_xor_u64(lo, st), oh = shfl_xor_u64(hi, st);
            lo = (lane & st) == 0 ? (ol < lo ? ol : lo) : (ol > lo ? ol : lo);
            hi = (lane & st) == 0 ? (oh < hi ? oh : hi) : (oh > hi ? oh : hi);
        }
        b[0] = lo;
        b[1] = hi;
    }
}

// Adds the keys of the lanes in m. A few keys go in one by one (a ballot
// gives the place, a shuffle shifts the rest: about 20 issue slots each);
// more are sorted across the warp and merged.
template <int KR>
__device__ __forceinline__ void list_add(uint64_t (&b)[KR], uint64_t key, unsigned m) {
    const int lane = threadIdx.x & 31;
    if (__popc(m) > kInsertMax) {
        list_merge<KR>(b, (m >> lane) & 1u ? key : kKeyMax);
        return;
    }
    while (m) {
        const uint64_t kx = __shfl_sync(kFullMask, key, __ffs(m) - 1);
        m &= m - 1;
        if constexpr (KR == 2) {  // the largest of the first register moves to the second
            uint64_t up = __shfl_up_sync(kFullMask, b[1], 1);
            const uint64_t last = __shfl_sync(kFullMask, b[0], 31);
            if (lane == 0) up = last;
            // elements above kx shift up by one; kx lands behind the last one below it
            b[1] = kx < b[1] ? (kx < up ? up : kx) : b[1];
        }
        uint64_t up = __shfl_up_sync(kFullMask, b[0], 1);
        if (lane == 0) up = 0;
        b[0] = kx < b[0] ? (kx < up ? up : kx) : b[0];
    }
}

// The element of rank r (0-based) of 32 * G values, G per lane.
template <int G>
__device__ __forceinline__ unsigned warp_rank_value(unsigned (&v)[G], int r) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int size = 2; size <= 32 * G; size <<= 1) {
#pragma unroll
        for (int st = size >> 1; st > 0; st >>= 1) {
            if (st == 32) {
                const unsigned a = v[0], c = v[G - 1];
                v[0] = min(a, c);
                v[G - 1] = max(a, c);
            } else {
#pragma unroll
                for (int j = 0; j < G; ++j) {
                    const unsigned o = __shfl_xor_sync(kFullMask, v[j], st);
                    const bool asc = ((j * 32 + lane) & size) == 0, lower = (lane & st) == 0;
                    v[j] = lower == asc ? min(v[j], o) : max(v[j], o);
                }
            }
        }
    }
    unsigned x = __shfl_sync(kFullMask, v[0], r & 31);
    if (G == 2 && r >= 32) x = __shfl_sync(kFullMask, v[G - 1], r & 31);
    return x;
}

// The bits of a list's k-th distance (all ones while it holds fewer than k
// keys), and the distance (+inf then).
template <int KR>
__device__ __forceinline__ unsigned list_kth_bits(const uint64_t (&b)[KR], int k) {
    return KR == 1 ? __shfl_sync(kFullMask, static_cast<unsigned>(b[0] >> 32), k - 1)
                   : __shfl_sync(kFullMask, static_cast<unsigned>(b[KR - 1] >> 32), k - 33);
}
template <int KR>
__device__ __forceinline__ float list_kth(const uint64_t (&b)[KR], int k) {
    const unsigned h = list_kth_bits<KR>(b, k);
    return h == 0xFFFFFFFFu ? inf_f() : __uint_as_float(h);
}

// Writes a finished row (whole warp) in the reference's slot order: the keys
// below the k-th by ascending index, then the ties (already in index order).
template <int KR>
__device__ __forceinline__ void emit_row(const uint64_t (&b)[KR], int k, int64_t n, unsigned self,
                                         int32_t* __restrict__ nbr_idx, float* __restrict__ nbr_d2,
                                         float* __restrict__ kdist2) {
    const int lane = threadIdx.x & 31;
    const unsigned kbits = KR == 1 ? __shfl_sync(kFullMask, static_cast<unsigned>(b[0] >> 32), k - 1)
                                   : __shfl_sync(kFullMask, static_cast<unsigned>(b[KR - 1] >> 32), k - 33);
    int below = 0, slot[KR];
    unsigned ix[KR];
#pragma unroll
    for (int j = 0; j < KR; ++j) {
        below += __popc(__ballot_sync(kFullMask, key_bits(b[j]) < kbits));  // all within the first k
        ix[j] = key_index(b[j]);
        slot[j] = 0;
    }
    for (int q = 0; q < below; ++q) {
        unsigned o = __shfl_sync(kFullMask, ix[0], q & 31);
        if (KR == 2 && q >= 32) o = __shfl_sync(kFullMask, ix[KR - 1], q & 31);
#pragma unroll
        for (int j = 0; j < KR; ++j) slot[j] += o < ix[j] ? 1 : 0;
    }
#pragma unroll
    for (int j = 0; j < KR; ++j) {
        const int e = 32 * j + lane;
        if (e < k) {
            const int64_t o = static_cast<int64_t>(e < below ? slot[j] : e) * n + self;
            nbr_idx[o] = static_cast<int32_t>(ix[j] & 0x7FFFFFFFu);
            nbr_d2[o] = __uint_as_float(key_bits(b[j]));
        }
    }
    if (lane == 0) kdist2[self] = __uint_as_float(kbits);
}

}  // namespace culof_gb300
