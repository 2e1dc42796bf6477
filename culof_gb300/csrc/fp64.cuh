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

// RN(a / b) of two floats, from y = RN(1 / b), once per b: q0 = RN(a y), r = a
// - q0 b, q = RN(q0 + r y), the correction of a quotient by one residual (P.
// Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34, 1990). With 24-bit significands q is the
// correctly rounded quotient: q0 is off by at most 1.5 ulp, so r has at most 25
// significant bits above ulp(q0) ulp(b) and is exact, and q0 + r y before its
// rounding is off from a / b by at most 2^-104 of it, while a / b, not a
// midpoint of two neighbouring doubles (a 54-bit midpoint M times b has more
// than 24 bits), is at least 2^-78 away from one. `quick`: y is neither zero
// nor infinite nor not a number (b is none of infinite, zero, not a number); an
// infinite a would leave r = inf - inf. The rest takes the division itself.
__device__ __forceinline__ bool quotient_quick(double y) {
    return fabs(y) < __longlong_as_double(0x7ff0000000000000ll) && y != 0.0;
}
__device__ __forceinline__ double quotient(float a, double b, double y, bool quick) {
    const double x = widen(a);
    if (quick && (__float_as_uint(a) & 0x7FFFFFFFu) < 0x7F800000u) {
        const double q0 = __dmul_rn(x, y);
        return __fma_rn(__fma_rn(-q0, b, x), y, q0);
    }
    return __ddiv_rn(x, b);
}

}  // namespace culof_gb300
