// Which of two forms of a product a call takes, decided on the device.
//
// A pair of fp16 values keeps 22 bits of a value down to 2^-17 of the largest of its scale's range
// and loses one more with every halving below (gemm_split.h); two TF32 values keep 21 bits
// anywhere. Where all values of a pixel, or all of a channel in some pixels, lie below 2^-16 of
// the largest, pairs would cost them precision that the fp32 interpolation still had (2^-24 of
// the largest value in the interpolation), so the TF32 form takes over. Both forms are launched and
// one returns at once: the host does not know the values, and asking for them would stop it.
#pragma once

#include <stdint.h>

namespace msda {

// What the layout kernels note of an operand with one or two factors: {largest magnitudes of the two,
// kLeastFrom minus the smallest nonzero maximum of a block of either}, as float bit patterns. Blocks:
// up to 32 or 64 channels of a pixel, 8 to 32 pixels of a channel. Zeros: nothing seen.
constexpr uint32_t kLeastFrom = 0x7f800000u;
constexpr int kPairSpread = 16;   // widest spread of block maxima, in powers of two, for pairs

struct RangeGate {
    const uint32_t* range[2];   // four words each; the first null: run always, the second may be null
    int if_wide;                // run where one of them spreads wider than kPairSpread (else where none)
};

#ifdef __CUDACC__
__device__ __forceinline__ bool range_is_wide(const uint32_t* range) {
    const uint4 w = *reinterpret_cast<const uint4*>(range);
    const int a = w.z == 0u ? 0 : static_cast<int>(w.x >> 23) - static_cast<int>((kLeastFrom - w.z) >> 23);
    const int b = w.w == 0u ? 0 : static_cast<int>(w.y >> 23) - static_cast<int>((kLeastFrom - w.w) >> 23);
    return a + b > kPairSpread;
}
// The same answer for every thread of a grid.
__device__ __forceinline__ bool gate_open(const RangeGate& g) {
    if (g.range[0] == nullptr) return true;
    const bool wide = range_is_wide(g.range[0]) || (g.range[1] != nullptr && range_is_wide(g.range[1]));
    return wide == (g.if_wide != 0);
}
#endif

}  // namespace msda
