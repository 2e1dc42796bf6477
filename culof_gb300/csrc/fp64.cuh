// Conversions between float and double with integer instructions: the same
// values as the conversion instructions, which take a slot of the FP64 unit
// each (one warp instruction per 64 cycles and scheduler on this GPU, where an
// addition costs the same).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace culof_gb300 {

// A normal float is widened by moving its fields (exponent bias 127 to 1023),
// a zero keeps its sign; the rest takes the conversion.
__device__ __forceinline__ double widen(float x) {
    const unsigned u = __float_as_uint(x), a = u & 0x7FFFFFFFu;
    if (a - 0x00800000u < 0x7F000000u)
        return __hiloint2double(static_cast<int>((u & 0x80000000u) | ((a >> 3) + (896u << 20))), static_cast<int>(u << 29));
    if (a == 0u) return __hiloint2double(static_cast<int>(u), 0);
    return static_cast<double>(x);
}

// Round to nearest even. A double whose exponent lies in a normal float's
// range keeps its upper 23 fraction bits, one more if the other 29 are over
// half, or half and the last kept bit odd (a carry moves into the exponent,
// past the largest float into infinity, as rounding does).
__device__ __forceinline__ float narrow(double x) {
    const unsigned hi = static_cast<unsigned>(__double2hiint(x)), lo = static_cast<unsigned>(__double2loint(x));
    const unsigned a = hi & 0x7FFFFFFFu;
    if (a - (897u << 20) < ((1151u - 897u) << 20)) {
        const unsigned kept = ((a - (896u << 20)) << 3) | (lo >> 29), rest = lo & 0x1FFFFFFFu;
        const unsigned up = rest + (kept & 1u) > 0x10000000u ? 1u : 0u;
        return __uint_as_float((hi & 0x80000000u) | (kept + up));
    }
    return __double2float_rn(x);
}

}  // namespace culof_gb300
