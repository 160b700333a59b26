// Conversions between FP64 and FP32 by integer operations on the bit patterns
// (internal linkage in each translation unit that includes this file).
#pragma once

#include <cuda_runtime.h>

namespace pg {
namespace {

// ---- FP64 inputs on the integer pipe -------------------------------------
// GB300's FP64 pipe is narrow (1/64 of FP32) and also runs the conversions
// between FP64 and FP32; these take the integer pipe.

// v rounded to FP32 (round half away from zero on the dropped bits: equal to
// round-to-nearest-even except on exact ties). Integer operations only:
// magnitudes below the FP32 normal range give a signed zero (flush to zero),
// above it a signed infinity; NaN stays NaN.
__device__ __forceinline__ float f64_to_f32(double v) {
    const unsigned hw = (unsigned)__double2hiint(v), lw = (unsigned)__double2loint(v);
    const unsigned sign = hw & 0x80000000u;
    const unsigned e = (hw >> 20) & 0x7FFu;
    const unsigned mag = ((((hw & 0x7FFFFFFFu) - (896u << 20)) << 3) | (lw >> 29)) +
                         ((lw >> 28) & 1u);
    const bool nan = e == 0x7FFu && ((hw & 0xFFFFFu) | lw) != 0u;
    const unsigned bits = e < 897u ? 0u : (e > 1150u ? (nan ? 0x7FC00000u : 0x7F800000u) : mag);
    return __uint_as_float(sign | bits);
}

// v = hi + lo: hi is v truncated to 24 significant bits, lo the remaining 29
// bits rounded to FP32 (|v - hi - lo| <= 2^-48 |v|) for 2^-74 <= |v| < 2^127;
// outside that range hi = f64_to_f32(v) and lo = 0. Integer operations only.
__device__ __forceinline__ float2 split_f64(double v) {
    const unsigned hw = (unsigned)__double2hiint(v), lw = (unsigned)__double2loint(v);
    const unsigned e = (hw >> 20) & 0x7FFu;
    const unsigned sign = hw & 0x80000000u;
    const float hi =
        __uint_as_float(sign | ((((hw & 0x7FFFFFFFu) - (896u << 20)) << 3) | (lw >> 29)));
    const unsigned rem = lw & 0x1FFFFFFFu;
    // the 29-bit remainder as (6 bits) 2^23 + (23 bits), each exact in FP32
    const float r_lo = __uint_as_float(0x4B000000u | (rem & 0x7FFFFFu)) - 8388608.f;
    const float r_hi = __uint_as_float(0x4B000000u | (rem >> 23)) - 8388608.f;
    const float r = fmaf(r_hi, 8388608.f, r_lo) * __uint_as_float(((e - 948u) & 0xFFu) << 23);
    const bool normal = e - 949u <= 200u;
    return make_float2(normal ? hi : f64_to_f32(v),
                       normal ? __uint_as_float(__float_as_uint(r) | sign) : 0.f);
}

// x exactly in FP64 (integer operations; FP32 subnormals give a signed zero)
__device__ __forceinline__ double f32_to_f64(float x) {
    const unsigned u = __float_as_uint(x);
    const unsigned sign = u & 0x80000000u;
    const unsigned ex = (u >> 23) & 0xFFu;
    const unsigned hw_n = sign | (((u & 0x7FFFFFFFu) >> 3) + (896u << 20));
    const unsigned hw_s = sign | 0x7FF00000u | ((u & 0x7FFFFFu) >> 3);  // inf, NaN
    const unsigned hw = ex == 0u ? sign : (ex == 0xFFu ? hw_s : hw_n);
    return __hiloint2double((int)hw, ex == 0u ? 0 : (int)(u << 29));
}

}  // namespace
}  // namespace pg
