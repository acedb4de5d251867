// Exponents of the fp16 pairs described in gemm_split.h.
#pragma once

#include <cuda_fp16.h>

#include "gemm_split.h"

namespace msda {

__device__ __forceinline__ float exp2_int(int e) { return __int_as_float((127 + e) << 23); }

// e with bound * 2^e < 2^15
__device__ __forceinline__ int split_exponent(const SplitScale& s, long long row) {
    const int E = static_cast<int>(s.bits[row * s.step] >> 23);
    const int e = s.bits2 == nullptr ? 141 - E : 266 - E - static_cast<int>(*s.bits2 >> 23);
    return max(-126, min(126, e));
}

// Bit pattern of |v|, 0 for Inf and NaN (they become Inf and NaN whatever the scale).
__device__ __forceinline__ uint32_t finite_magnitude(float v) {
    const uint32_t b = __float_as_uint(v) & 0x7fffffffu;
    return b < 0x7f800000u ? b : 0u;
}

// Two values times `s` as {hi pair, lo pair}.
__device__ __forceinline__ uint2 split_pair(float x, float y, float s) {
    x *= s;
    y *= s;
    const __half2 hi = __floats2half2_rn(x, y);
    const float2 h = __half22float2(hi);
    const __half2 lo = __floats2half2_rn(x - h.x, y - h.y);
    return make_uint2(*reinterpret_cast<const uint32_t*>(&hi), *reinterpret_cast<const uint32_t*>(&lo));
}

}  // namespace msda
