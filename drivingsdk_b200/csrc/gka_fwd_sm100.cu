// Geometric kernel attention forward for sm_100a: out[b,q,h,:] = sum over (level, point) of
// attention * value[b, level, clamp(y), clamp(x), h, :] — integer pixel coordinates, clamped
// into the level, no interpolation. Replaces the reference's device kernel
// (kernels/geometric_kernel_attention/op_kernel/geometric_kernel_attention.cpp:123-182).
// Two forms: a map in shared memory (below), and the same kernel template as the bilinear
// operator with one row per sample instead of four.
#include "msda_bwd_sorted.cuh"   // level table of a CTA
#include "msda_fwd_kernel.cuh"

namespace msda {

constexpr size_t kMapSmem = 224 * 1024;   // most for the map and the records

// Value of one (batch, head) in shared memory, or a slice of its channels if the map is large,
// where its rows arrive at twice the 64 bytes per clock and SM that loads through L1 return,
// which is what bounds the other form (24 x 7156 x 4 tasks of 15 rows of 256 bytes, 15 x 25
// pixels: 227 -> 131 us, 238 -> 115 us in bf16).
//
// The CTAs share the (batch, head, slice, query) tasks in equal consecutive ranges; where a range
// crosses into the next map, the CTA loads that. 32 / LPR tasks per warp at a time: records
// (row, weight) of all their samples first, lane = sample; then a group of LPR lanes walks one
// task, each lane 16 bytes of the row (of its slice).
template <typename T, int LPR>
__global__ void __launch_bounds__(1024, 1)
gka_map_fwd_kernel(const __grid_constant__ Params p, const uint32_t slices, const FastDiv fd_p) {
    constexpr int VEC = Elem<T>::kVec;
    constexpr uint32_t TASKS = 32 / LPR;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ SortLevels lv;
    if (!load_sort_levels(p, lv)) {
        clear_output<T>(p);
        return;
    }
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const uint32_t g = lane / LPR, j = lane % LPR;
    const uint32_t Q = p.Q, H = p.H, LP = p.LP;
    const uint32_t stride = LP | 1u;   // odd: the tasks' records lie in different banks
    const uint32_t pieces = static_cast<uint32_t>(p.K) * LPR;
    uint2* recs = reinterpret_cast<uint2*>(smem + pieces * 16u) + warp * TASKS * stride;
    const unsigned char* row_j = smem + j * 16u;
    const T* loc = static_cast<const T*>(p.loc);
    const T* attn = static_cast<const T*>(p.attn);
    T* out = static_cast<T*>(p.out);

    const uint64_t tasks = static_cast<uint64_t>(p.ntasks) * slices;
    uint64_t n = tasks * blockIdx.x / gridDim.x;
    const uint64_t end = tasks * (blockIdx.x + 1) / gridDim.x;
    while (n < end) {
        const uint32_t map = static_cast<uint32_t>(n / Q), slice = map % slices;
        const uint32_t b = map / slices / H, h = map / slices - b * H;
        const uint32_t q0 = static_cast<uint32_t>(n - static_cast<uint64_t>(map) * Q);
        const uint32_t q1 = static_cast<uint32_t>(min(static_cast<uint64_t>(Q), q0 + (end - n)));
        n += q1 - q0;
        const uint4* value = static_cast<const uint4*>(p.value) +
                             (static_cast<size_t>(b) * p.K * H + h) * p.pieces + slice * LPR;
        __syncthreads();   // the map before is no longer read
        for (uint32_t i = threadIdx.x; i < pieces; i += blockDim.x)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem + i * 16u)),
                         "l"(value + static_cast<size_t>(i / LPR) * H * p.pieces + i % LPR)
                         : "memory");
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();

        for (uint32_t q = q0 + warp * TASKS; q < q1; q += warps * TASKS) {
            const uint32_t count = min(TASKS, q1 - q);
            const size_t first = (static_cast<size_t>(b) * Q + q) * H + h;   // task
#pragma unroll 2
            for (uint32_t i = lane; i < count * LP; i += 32) {
                const uint32_t task = fd_div(i, p.fd_lp), s = i - task * LP;
                const size_t gi = (first + static_cast<size_t>(task) * H) * LP + s;
                const float2 xy = load_pair(loc + 2 * gi);
                const float4 geo = lv.geo[fd_div(s, fd_p)];
                const int W = __float_as_int(geo.z);
                const int x = min(max(__float2int_rz(xy.x), 0), W - 1);
                const int y = min(max(__float2int_rz(xy.y), 0), __float2int_rz(geo.y) - 1);
                uint32_t row = __float_as_uint(geo.w) + static_cast<uint32_t>(y * W + x);
#ifdef MSDA_DEBUG_BOUNDS
                if (row >= static_cast<uint32_t>(p.K)) {
                    atomicOr(p.status, kStatusOutOfBounds);
                    row = 0u;
                }
#endif
                recs[task * stride + s] =
                    make_uint2(row * (LPR * 16u), __float_as_uint(Elem<T>::to_f(__ldg(attn + gi))));
            }
            __syncwarp();
            if (g < count) {
                f32x2 sum[VEC / 2];
#pragma unroll
                for (int e = 0; e < VEC / 2; ++e) sum[e] = 0ull;
                const uint2* rec = recs + g * stride;
#pragma unroll 5
                for (uint32_t s = 0; s < LP; ++s) {
                    const uint2 r = rec[s];
                    const uint4 raw = *reinterpret_cast<const uint4*>(row_j + r.x);
                    const f32x2 w2 = pack2(__uint_as_float(r.y), __uint_as_float(r.y));
                    float f[VEC];
                    unpack16<T>(raw, f);
#pragma unroll
                    for (int e = 0; e < VEC / 2; ++e)
                        sum[e] = fma2(w2, pack2(f[2 * e], f[2 * e + 1]), sum[e]);
                }
                float f[VEC];
#pragma unroll
                for (int e = 0; e < VEC / 2; ++e) {
                    const float2 v = unpack2(sum[e]);
                    f[2 * e] = v.x;
                    f[2 * e + 1] = v.y;
                }
                *reinterpret_cast<uint4*>(out + (first + static_cast<size_t>(g) * H) * p.D +
                                          (slice * LPR + j) * VEC) = pack16<T>(f);
            }
            __syncwarp();   // the records are read
        }
    }
}

// `taken` false: the sizes are for something else.
template <typename T, int LPR>
static cudaError_t launch_map_fwd(const Params& p, const LaunchShape& ls, cudaStream_t stream, bool* taken) {
    *taken = false;
    if (p.pieces % LPR != 0) return cudaSuccess;
    auto kern = gka_map_fwd_kernel<T, LPR>;
    const uint32_t slices = static_cast<uint32_t>(p.pieces / LPR);
    // four narrow slices are slower than gathering whole rows (12 x 5000 x 8 tasks of 15 rows of 256
    // bytes, 2250 pixels: 212 against 179 us)
    if (slices > 3) return cudaSuccess;
    const size_t map = static_cast<size_t>(p.K) * LPR * 16;
    const size_t record = static_cast<size_t>(32 / LPR) * (p.LP | 1) * sizeof(uint2);   // of a warp
    // two CTAs of 16 warps per SM, or one of 32, or of 16 if that leaves too little room
    const bool two = 2 * (map + 16 * record) <= kMapSmem;
    const int threads = (two || map + 32 * record > kMapSmem) ? 512 : 1024;
    const size_t smem = map + threads / 32 * record;
    if (smem > kMapSmem) return cudaSuccess;
    // Every CTA and every map has its rows loaded once more. That pays from some three samples per
    // loaded row on, two in 16 bits (24 x 204 x 4 tasks of 15 samples, 375 pixels of 256 bytes: 3.2 and
    // 10.8 against 11.7 us, 2.2 and 9.8 against 9.6; bf16 2.2 and 10.0 against 11.3, 1.2 and 8.3
    // against 8.1).
    constexpr int kLeast = sizeof(T) == 4 ? 3 : 2;
    const long long grid = static_cast<long long>(ls.sm_count) *
                           (ls.ctas_per_sm > 0 ? ls.ctas_per_sm : two ? 2 : 1);
    const long long maps = static_cast<long long>(p.B) * p.H * slices;
    if (p.ntasks * slices * p.LP < kLeast * (grid + maps) * p.K) return cudaSuccess;
    int resident = 0;   // (asked for the shared-memory limit that the call sets)
    const cudaError_t e = resident_ctas(reinterpret_cast<const void*>(kern), threads, smem, &resident);
    if (e != cudaSuccess) return e;
    *taken = true;
    kern<<<static_cast<unsigned>(grid), threads, smem, stream>>>(p, slices,
                                                                 make_fastdiv(static_cast<uint32_t>(p.P)));
    return cudaGetLastError();
}

// The widest slices that fit: each slice reads locations and weights again.
template <typename T>
static cudaError_t launch_map_fwd_typed(const Params& p, const RowPlan& rp, const LaunchShape& ls,
                                        cudaStream_t stream, bool* taken) {
    *taken = false;
    if (rp.scalar || reinterpret_cast<uintptr_t>(p.loc) % (2 * sizeof(T)) != 0) return cudaSuccess;
    cudaError_t e = launch_map_fwd<T, 16>(p, ls, stream, taken);
    if (e == cudaSuccess && !*taken) e = launch_map_fwd<T, 8>(p, ls, stream, taken);
    if (e == cudaSuccess && !*taken) e = launch_map_fwd<T, 4>(p, ls, stream, taken);
    return e;
}

cudaError_t launch_gka_forward(const Params& p, int dtype, const RowPlan& rp,
                               const LaunchShape& ls, cudaStream_t stream) {
    bool taken = false;
    cudaError_t e = cudaErrorInvalidValue;
    switch (dtype) {
        case 0: e = launch_map_fwd_typed<float>(p, rp, ls, stream, &taken); break;
        case 1: e = launch_map_fwd_typed<__half>(p, rp, ls, stream, &taken); break;
        case 2: e = launch_map_fwd_typed<__nv_bfloat16>(p, rp, ls, stream, &taken); break;
        default: break;
    }
    if (e != cudaSuccess || taken) return e;
    return launch_forward_cps<1>(p, dtype, rp, ls, stream);
}

}  // namespace msda
