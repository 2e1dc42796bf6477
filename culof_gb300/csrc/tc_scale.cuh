// What a tensor-path call starts from on the device: the f16 scale of its operands
// and the counts of its lost rows' groups.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "fast.cuh"
#include "prep.cuh"
#include "sweep_common.cuh"

namespace culof_gb300 {

// Scale record on the device: sc = 2^S, k2 = -2 * 2^-2S (undoes the scale of
// a Gram value and doubles it), eta = 2^-14 * 2^-S (absolute f16 rounding
// bound in unscaled units), all = 1 when the filter is disabled, resmax the
// largest residual norm (tc_resid_kernel).
struct TcScale {
    float sc, k2, eta, all;
    unsigned resmax;  // float bits
};

// One warp: the scale exponent from the features' ranges. The filter is off if
// f = |b|^2 - 2 a.b could overflow: |f| <= 3 nmax (1 + 2^-8) and the bounds add
// 2 m0 + slack, less than nmax, which together stay below 2^127 up to nmax =
// 2^124 = kMaxFilterNorm (the comparison also catches a norm that is not a number).
__device__ __forceinline__ void tc_scale_record(const unsigned* __restrict__ mm, int d,
                                                const unsigned* __restrict__ max_norm_bits, TcScale* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    float mx = 0.0f;
    bool finite = __uint_as_float(*max_norm_bits) <= sweep::kMaxFilterNorm;
    for (int f = lane; f < d; f += 32) {
        const float lo = range_lo(mm, f), hi = range_hi(mm, f);
        finite = finite && isfinite(lo) && isfinite(hi);
        mx = fmaxf(mx, fmaxf(fabsf(lo), fabsf(hi)));
    }
    mx = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mx)));
    finite = __all_sync(0xffffffffu, finite);
    if (lane != 0) return;
    int S = 0;
    bool all = !finite;
    if (finite && mx > 0.0f) {
        S = 14 - ilogbf(mx);
        if (S > 62 || S < -62) all = true;
    }
    if (all) S = 0;
    TcScale r;
    r.sc = ldexpf(1.0f, S);
    r.k2 = -ldexpf(1.0f, 1 - 2 * S);
    r.eta = ldexpf(1.0f, -14 - S);
    r.all = all ? 1.0f : 0.0f;
    r.resmax = 0u;
    *out = r;
}

// (16-byte aligned)
struct TcStart {
    TcScale scale;
    unsigned pad[3];
    int arrived[kLostGroups];
};

// One warp.
__device__ __forceinline__ void tc_start(const unsigned* __restrict__ mm, int d, const unsigned* __restrict__ max_norm_bits,
                                         TcStart* __restrict__ out) {
    for (int i = threadIdx.x & 31; i < kLostGroups; i += 32) out->arrived[i] = 0;
    tc_scale_record(mm, d, max_norm_bits, &out->scale);
}

}  // namespace culof_gb300
