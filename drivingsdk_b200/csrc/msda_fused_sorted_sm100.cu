// Fused operator, backward over cell-sorted samples, for sm_100a. Where sorting pays (sort_pays in
// msda_capi.cu) the sorted backward of the bilinear operator does the work, between two kernels that
// take 9 and 12 ps per sample (about 20 bytes of memory each, and the reductions over a task):
//   fused_samples_kernel     reference points, offsets and logits -> locations and weights, in fp32 as the
//                            other fused kernels keep them in registers
//   fused_gradients_kernel   gradients of locations and weights -> of offsets, logits and reference points
#include "msda_bwd_sorted.cuh"
#include "msda_tile.cuh"

namespace msda {

// One lane per sample: use(whether the lane has one, its task, global sample number, task in the item,
// sample in the task, what load(task, sample number) gave) by all lanes of a warp. An item is loaded
// while the one before it is used.
template <typename Load, typename Use>
__device__ __forceinline__ void for_each_item(const Params& p, int warp, int lane, const Load& load, const Use& use) {
    int tl, s;
    lane_sample_index(p, 0, lane, tl, s);
    const bool mine = tl < p.tasks_per_item && s < p.LP;
    ItemWalk walk = make_walk(p, warp);
    auto task = [&](long long idx) { return idx * p.tasks_per_item + tl; };
    auto active = [&](long long idx) { return mine && idx < walk.end && task(idx) < p.ntasks; };
    decltype(load(0ll, 0ll)) now{}, next{};
    if (active(walk.idx)) now = load(task(walk.idx), task(walk.idx) * p.LP + s);
    for (; walk.idx < walk.end; walk.idx += walk.stride) {
        const long long t = task(walk.idx), after = task(walk.idx + walk.stride);
        if (active(walk.idx + walk.stride)) next = load(after, after * p.LP + s);
        use(active(walk.idx), t, t * p.LP + s, tl, s, now);
        __syncwarp();   // the scratch is used again
        now = next;
    }
}

template <typename T>
__global__ void __launch_bounds__(kThreadsPerCta)
fused_samples_kernel(const __grid_constant__ Params p, float2* __restrict__ loc, float* __restrict__ prob) {
    __shared__ float s_scratch[kWarpsPerCta][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    bool ok;
    const LaneLevels lv = load_lane_levels(p, lane, ok);
    if (!ok) return;   // the sort refuses the table too
    const T* off = static_cast<const T*>(p.loc);
    const T* logit = static_cast<const T*>(p.attn);
    struct Raw {
        float a, x, y, ref_x, ref_y;
    };
    auto load = [&](long long t, long long gi) {
        const T* ref = static_cast<const T*>(p.ref) +
                       (static_cast<size_t>(fd_div(static_cast<uint32_t>(t), p.fd_h)) * p.L + lv.level0) * 2;
        return Raw{Elem<T>::to_f(logit[gi]), Elem<T>::to_f(off[2 * gi]), Elem<T>::to_f(off[2 * gi + 1]),
                   Elem<T>::to_f(ref[0]), Elem<T>::to_f(ref[1])};
    };
    for_each_item(p, warp, lane, load, [&](bool active, long long, long long gi, int tl, int, const Raw& r) {
        const float a = active ? r.a : -INFINITY;
        const float m = task_max(p, a, lane, tl, s_scratch[warp]);
        const float e = active ? __expf(a - m) : 0.f;
        const float sum = task_sum(p, e, lane, tl, s_scratch[warp]);
        if (active) {
            loc[gi] = make_float2(r.ref_x + r.x / static_cast<float>(lv.w0), r.ref_y + r.y / static_cast<float>(lv.h0));
            prob[gi] = e / sum;
        }
    });
}

// grad_loc / grad_attn may be p.grad_loc / p.grad_attn themselves (fp32): every sample is read and
// written by the same lane.
template <typename T>
__global__ void __launch_bounds__(kThreadsPerCta)
fused_gradients_kernel(const __grid_constant__ Params p, const float* __restrict__ prob, const float2* grad_loc,
                       const float* grad_attn) {
    __shared__ float s_scratch[kWarpsPerCta][96];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* scratch = s_scratch[warp];
    bool ok;
    const LaneLevels lv = load_lane_levels(p, lane, ok);
    if (!ok) return;
    struct Raw {
        float2 g;
        float a, pr;
    };
    auto load = [&](long long, long long gi) { return Raw{grad_loc[gi], grad_attn[gi], prob[gi]}; };
    for_each_item(p, warp, lane, load, [&](bool active, long long t, long long gi, int tl, int s, const Raw& r) {
        const float2 g = active ? r.g : make_float2(0.f, 0.f);
        const float a = active ? r.a : 0.f, pr = active ? r.pr : 0.f;
        // softmax: d logit_s = p_s * (d a_s - sum_j p_j * d a_j)
        const float dot = task_sum(p, pr * a, lane, tl, scratch);
        scratch[32 + lane] = g.x;
        scratch[64 + lane] = g.y;
        __syncwarp();
        if (!active) return;
        store_pair(static_cast<T*>(p.grad_loc) + 2 * gi, g.x / static_cast<float>(lv.w0),
                   g.y / static_cast<float>(lv.h0));
        static_cast<T*>(p.grad_attn)[gi] = Elem<T>::from_f(pr * (a - dot));
        if (s % p.P == 0) {
            // first point of a level: the reference point gets the sum over this head's points
            float sx = 0.f, sy = 0.f;
            for (int i = 0; i < p.P; ++i) {
                sx += scratch[32 + lane + i];
                sy += scratch[64 + lane + i];
            }
            float* to = p.grad_ref +
                        (static_cast<size_t>(fd_div(static_cast<uint32_t>(t), p.fd_h)) * p.L + lv.level0) * 2;
            atomicAdd(to, sx);
            atomicAdd(to + 1, sy);
        }
    });
}

template <typename T>
static cudaError_t launch_fused_sorted_typed(const Params& p, const SortParams& sp, const FusedSamples& fs,
                                             const LaunchShape& ls, cudaStream_t stream) {
    int grid = 0;
    auto before = fused_samples_kernel<T>;
    cudaError_t e = persistent_grid(reinterpret_cast<const void*>(before), 0, LaunchShape{ls.sm_count, 0}, p, &grid);
    if (e != cudaSuccess) return e;
    before<<<grid, kThreadsPerCta, 0, stream>>>(p, fs.loc, fs.prob);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;

    Params q = p;   // the bilinear operator's
    q.loc = fs.loc;
    q.attn = fs.prob;
    q.grad_loc = fs.grad_loc;
    q.grad_attn = fs.grad_attn;
    if constexpr (sizeof(T) == 4) e = launch_backward_sorted(q, sp, 0, ls, stream);
    else e = launch_sorted_bilinear<T, float>(q, sp, ls, stream);
    if (e != cudaSuccess) return e;

    auto after = fused_gradients_kernel<T>;
    e = persistent_grid(reinterpret_cast<const void*>(after), 0, LaunchShape{ls.sm_count, 0}, p, &grid);
    if (e != cudaSuccess) return e;
    after<<<grid, kThreadsPerCta, 0, stream>>>(p, fs.prob, fs.grad_loc, fs.grad_attn);
    return cudaGetLastError();
}

cudaError_t launch_fused_backward_sorted(const Params& p, const SortParams& sp, const FusedSamples& fs, int dtype,
                                         const LaunchShape& ls, cudaStream_t stream) {
    switch (dtype) {
        case 0: return launch_fused_sorted_typed<float>(p, sp, fs, ls, stream);
        case 1: return launch_fused_sorted_typed<__half>(p, sp, fs, ls, stream);
        case 2: return launch_fused_sorted_typed<__nv_bfloat16>(p, sp, fs, ls, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace msda
