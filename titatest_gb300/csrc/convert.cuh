// Conversions between FP32 and FP64 outside the FP64 pipe.
#pragma once

#include "cplx.cuh"

namespace crgpu {

// float <-> double by their bit fields: the conversion instructions share the
// FP64 pipe (2 lanes a cycle and SM).  Equal to the casts for every value;
// subnormals are met in earnest (potentials far from an electrode at large
// wavenumbers).  Infinities and NaN take the instruction, in a call: inlined,
// the compiler makes it unconditional and selects.
static __device__ __noinline__ double widen_any(float v) { return (double)v; }
static __device__ __noinline__ float narrow_any(double v) { return (float)v; }

__device__ __forceinline__ double widen(float v) {
    const unsigned b = __float_as_uint(v), s = b & 0x80000000u, e = (b >> 23) & 255u;
    unsigned m = b & 0x7fffffffu;
    if (e == 255u) return widen_any(v);
    unsigned ex = 896u << 20;
    if (e == 0u) {
        if (m == 0u) return __hiloint2double((int)s, 0);
        const int z = __clz((int)m) - 8;  // to the normal position
        m <<= z;
        ex -= (unsigned)z << 20;  // the leading bit adds one binade: exponent 1 - z
    }
    return __hiloint2double((int)(s | ((m >> 3) + ex)), (int)(m << 29));
}
// (float)v, to nearest even
__device__ __forceinline__ float narrow(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const unsigned e = (unsigned)(b >> 52) & 2047u, s = (unsigned)(b >> 32) & 0x80000000u;
    if (e >= 1150u) return narrow_any(v);  // the floats' last binade and beyond
    if (e < 897u) {                        // a subnormal or zero
        if (e < 872u) return __uint_as_float(s);
        const unsigned sh = 926u - e;  // 30 .. 54
        const unsigned long long m = (b & 0xfffffffffffffull) | (1ull << 52), r = m >> sh, rem = m & ((1ull << sh) - 1ull),
                                 half = 1ull << (sh - 1u);
        return __uint_as_float(s | ((unsigned)r + (rem > half || (rem == half && (r & 1ull)) ? 1u : 0u)));
    }
    unsigned long long t = (b & 0x7fffffffffffffffull) - (896ull << 52);
    t += 0x0fffffffull + ((t >> 29) & 1ull);
    return __uint_as_float((unsigned)(t >> 29) | s);
}
__device__ __forceinline__ double2 widen(float2 v) { return cz(widen(v.x), widen(v.y)); }
__device__ __forceinline__ float2 narrow(double2 v) { return cf(narrow(v.x), narrow(v.y)); }

}  // namespace crgpu
