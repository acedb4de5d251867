// The sampling halves of the deformable convolution, for dcn_split_sm100.cu. p.x, p.offset and p.mask
// as channels-last fp32 with whole quads of channels, 16-byte aligned. Return an msda_status.
#pragma once

#include <cuda_runtime.h>

#include "dcn_common.cuh"
#include "gemm_split.h"

namespace dcn {
// p.columns: the gradient of the columns; adds into p.grad_x, writes p.grad_offset and p.grad_mask.
// Pixel by pixel (dcn_sm100.cu).
int launch_scatter(const DcnParams& p, int sm_count, cudaStream_t stream);

// The grad_weight product from fp32 operands (dcn_sm100.cu).
int launch_weight_product(const float* grad_out, const float* columns, float* grad_weight, const dcn_shape* s,
                          const Derived& d, int sms, int* status_word, cudaStream_t stream);

// Over cell-sorted samples (dcn_sorted_sm100.cu), in a workspace of sorted_bytes() (0 where the form
// does not apply). The gather sorts, and writes the columns as fp16 pairs; the scatter reads what a
// gather of the same samples left in the workspace, and counts in *ticket, which must be zero (a
// counter of its own: backward passes over one forward may run at the same time). columns_f32 may
// be null.
size_t sorted_bytes(const dcn_shape* s, const Derived& d);
int launch_gather_sorted(const DcnParams& p, void* workspace, long long M, int N, uint16_t* columns,
                         size_t plane, const msda::SplitScale& bound, float* columns_f32, int sm_count,
                         cudaStream_t stream);
int launch_scatter_sorted(const DcnParams& p, const void* sorted, uint32_t* ticket, long long M, int N,
                          int sm_count, cudaStream_t stream);
}  // namespace dcn
