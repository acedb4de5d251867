// The scatter half of the deformable convolution's backward (dcn_sm100.cu), for dcn_split_sm100.cu.
#pragma once

#include <cuda_runtime.h>

namespace dcn {
struct DcnParams;
// p.columns: the gradient of the columns; adds into p.grad_x, writes p.grad_offset and p.grad_mask.
// Channels in whole quads, rows 16-byte aligned. Returns an msda_status.
int launch_scatter(const DcnParams& p, int sm_count, cudaStream_t stream);
}  // namespace dcn
