// Matrix products over operands that their producers have already split into fp16 pairs.
//
// An fp32 value v of an operand is stored as hi + lo of v * 2^e: hi = fp16(v * 2^e), lo =
// fp16(v * 2^e - hi), in two planes. e is chosen per row of the operand (or for all of it) from a
// bound on its magnitudes so that v * 2^e < 2^15; the pair then keeps 22 bits of v down to 2^-17
// of that bound and 2^-40 of it in absolute terms below (a TF32 pair keeps 21). Three products
// (lo*hi + hi*lo + hi*hi) at the fp16 rate give fp32-class accuracy at twice the rate of the
// three TF32 products of gemm_tc_sm100.cu, whose shared-memory traffic also includes splitting
// every tile. That accuracy is relative to the scale: a row (or, under one scale, a pixel) all of whose
// values lie far below it loses it, at 2^-30 all but 10 bits. Callers whose operands may spread that
// wide choose by range_gate.h.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "range_gate.h"

namespace msda {

// Where a row's bound comes from: bits[row * step] is the bit pattern of the largest finite
// magnitude; bits2 (optional) of a second factor of the values.
struct SplitScale {
    const uint32_t* bits;
    int step;
    const uint32_t* bits2;
};

struct SplitOperand {
    const uint16_t* hi;      // fp16; element (row, k) at hi[row * row_stride + k * k_stride]
    long long row_stride, k_stride;   // one of them is 1, the other a multiple of 8
    long long plane;         // lo = hi + plane, a multiple of 8
    SplitScale scale;        // by row
};

// C(m, n) (+)= sum_k A(m, k) * B(n, k) (+ bias[n]): fp32, row stride ldc. Both operands with k
// contiguous, or both with the row index contiguous; 16-byte aligned. `splits` > 1 cuts K into
// parts that are added into C (which must be zero before). Row-contiguous operands are read in
// blocks of 64 rows: up to 126 bytes past the last row of the last k must be readable.
cudaError_t gemm_split(const SplitOperand& A, const SplitOperand& B, float* C, long long ldc,
                       const float* bias, int M, int N, int K, int splits, const RangeGate& gate,
                       int* status_word, cudaStream_t stream);

}  // namespace msda
