// Geometric kernel attention backward over pixel-sorted samples for sm_100a
// (msda_bwd_sorted.cuh with one row per sample), all types.
#include "msda_bwd_sorted.cuh"

namespace msda {

cudaError_t launch_gka_backward_sorted(const Params& p, const SortParams& sp, int dtype,
                                       const LaunchShape& ls, cudaStream_t stream) {
    switch (dtype) {
        case 0: return launch_sorted_nearest<float>(p, sp, ls, stream);
        case 1: return launch_sorted_nearest<__half>(p, sp, ls, stream);
        case 2: return launch_sorted_nearest<__nv_bfloat16>(p, sp, ls, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace msda
