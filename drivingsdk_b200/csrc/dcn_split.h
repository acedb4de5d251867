// The sampling halves of the deformable convolution, for dcn_split_sm100.cu. p.x, p.offset and p.mask
// as channels-last fp32 with whole quads of channels, 16-byte aligned. Return an msda_status.
#pragma once

#include <cuda_runtime.h>

#include "dcn_common.cuh"
#include "gemm_split.h"

namespace dcn {
// Where the columns go: as fp16 pairs under one scale, or in fp32 where the values spread too wide for
// pairs (the same memory will do), or both.
struct ColumnsOut {
    uint16_t* pairs;
    size_t plane;            // halves per plane of the pairs
    float* f32;
    int keep_f32;            // in fp32 in any case
    msda::SplitScale bound;
    const uint32_t* range;   // range_gate.h
};

// p.columns: the gradient of the columns; adds into p.grad_x, writes p.grad_offset and p.grad_mask.
// Pixel by pixel (dcn_sm100.cu).
int launch_scatter(const DcnParams& p, int sm_count, cudaStream_t stream);

// The products of the forward and of grad_weight from fp32 operands (dcn_sm100.cu). With a gate, the
// caller has zeroed the result if weight_splits() or forward_splits() cuts the product.
int launch_forward_product(const float* columns, const float* weight, const float* bias, float* out,
                           const dcn_shape* s, const Derived& d, int sms, const msda::RangeGate& gate,
                           int* status_word, cudaStream_t stream);
int launch_weight_product(const float* grad_out, const float* columns, float* grad_weight, const dcn_shape* s,
                          const Derived& d, int sms, const msda::RangeGate& gate, int* status_word,
                          cudaStream_t stream);

// Over cell-sorted samples (dcn_sorted_sm100.cu), in a workspace of sorted_bytes() (0 where the form
// does not apply). The gather sorts, and writes the columns; the scatter reads what a
// gather of the same samples left in the workspace, and counts in *ticket, which must be zero (a
// counter of its own: backward passes over one forward may run at the same time).
size_t sorted_bytes(const dcn_shape* s, const Derived& d);
int launch_gather_sorted(const DcnParams& p, void* workspace, long long M, int N, const ColumnsOut& to,
                         int sm_count, cudaStream_t stream);
int launch_scatter_sorted(const DcnParams& p, const void* sorted, uint32_t* ticket, long long M, int N,
                          int sm_count, cudaStream_t stream);
}  // namespace dcn
