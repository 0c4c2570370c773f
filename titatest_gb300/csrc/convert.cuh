// Conversions between FP32 and FP64 outside the FP64 pipe.
#pragma once

#include "cplx.cuh"

namespace crgpu {

// float <-> double by their bit fields: the conversion instructions share the
// FP64 pipe (2 lanes a cycle and SM).  Exact as (double)v; zeros, subnormals,
// infinities and NaN take the instruction.
__device__ __forceinline__ double widen(float v) {
    const unsigned b = __float_as_uint(v), e = (b >> 23) & 255u;
    if (e - 1u >= 254u) return (double)v;
    return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(b << 29));
}
// (float)v, to nearest even
__device__ __forceinline__ float narrow(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    const unsigned e = (unsigned)(b >> 52) & 2047u;
    if (e - 897u >= 253u) return (float)v;  // outside the normal floats below their last binade
    unsigned long long t = (b & 0x7fffffffffffffffull) - (896ull << 52);
    t += 0x0fffffffull + ((t >> 29) & 1ull);
    return __uint_as_float((unsigned)(t >> 29) | ((unsigned)(b >> 32) & 0x80000000u));
}
__device__ __forceinline__ double2 widen(float2 v) { return cz(widen(v.x), widen(v.y)); }
__device__ __forceinline__ float2 narrow(double2 v) { return cf(narrow(v.x), narrow(v.y)); }

}  // namespace crgpu
