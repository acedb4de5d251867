// Parameters of the deformable-aggregation kernels (da_sm100.cu, da_sorted_sm100.cu).
#pragma once

#include "msda_launch.h"

namespace msda {

constexpr int kDaMaxMaps = 64;   // cams * scales
constexpr int kDaMaxGroups = 32;

struct DaParams {
    const float* feat;
    const float* loc;
    const float* wts;
    float* out;
    const float* grad_out;
    float* grad_feat;
    float* grad_loc;
    float* grad_wts;
    const int* shapes_dev;   // [cams*scales*2] (h, w), used when use_table == 0
    const int* starts_dev;   // [cams*scales]
    int use_table;
    int B, F, C, A, Pts, cams, scales, G;
    int S;         // samples per (batch, anchor): Pts * cams * scales
    int ppt;       // points per task: floor(32 / scales)
    int nparts;    // blocks of points: ceil(Pts / ppt)
    int cpg;       // channels per group
    uint32_t row_units;
    uint32_t warp_smem;
    long long ntasks;   // B * cams * nparts * A
    int lv_h[kDaMaxMaps], lv_w[kDaMaxMaps], lv_start[kDaMaxMaps];
};

// Backward over cell-sorted samples; dtype: type of feat, loc, wts and grad_out (the gradients are
// fp32). grad_feat, grad_loc and grad_wts must be zero before.
cudaError_t launch_da_backward_sorted(const DaParams& p, SortParams sp, int dtype, int sm_count,
                                      cudaStream_t stream);

}  // namespace msda
