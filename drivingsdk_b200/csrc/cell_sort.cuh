// Counting sort of samples by the cell of the map they fall into, and what the kernels that walk
// the sorted samples share: the backward of the attention operators (msda_bwd_sorted.cuh) and of
// deformable aggregation (da_sorted_sm100.cu).
#pragma once

#include <type_traits>

#include "msda_common.cuh"
#include "msda_launch.h"

namespace msda {

constexpr int kSortThreads = 1024;
constexpr uint32_t kSortCells = 24 * 1024;   // counters of one CTA: 96 KB, two CTAs per SM
constexpr uint32_t kMaxStream = 256;         // most consecutive sorted samples in one stream

template <typename TL>
__device__ __forceinline__ float2 load_pair(const TL* p);
template <>
__device__ __forceinline__ float2 load_pair<float>(const float* p) {
    return __ldg(reinterpret_cast<const float2*>(p));
}
template <>
__device__ __forceinline__ float2 load_pair<__half>(const __half* p) {
    return __half22float2(__ldg(reinterpret_cast<const __half2*>(p)));
}
template <>
__device__ __forceinline__ float2 load_pair<__nv_bfloat16>(const __nv_bfloat16* p) {
    const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(p));
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}

// The sample's cell in its level, or kNoRow for a sample that takes no part.
template <int CPS>
__device__ __forceinline__ uint32_t sample_cell(float2 xy, int W, int H) {
    if constexpr (CPS == 4) {
        const float wf = static_cast<float>(W), hf = static_cast<float>(H);
        const float x = xy.x * wf - 0.5f;
        const float y = xy.y * hf - 0.5f;
        if (!((x > -1.f) && (y > -1.f) && (x < wf) && (y < hf))) return kNoRow;
        return static_cast<uint32_t>(__float2int_rd(y) + 1) * static_cast<uint32_t>(W + 1) +
               static_cast<uint32_t>(__float2int_rd(x) + 1);
    } else {
        const int x = min(max(__float2int_rz(xy.x), 0), W - 1);
        const int y = min(max(__float2int_rz(xy.y), 0), H - 1);
        return static_cast<uint32_t>(y * W + x);
    }
}

// Counters in the shared memory of CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_address(const uint32_t* p, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_count(uint32_t addr) {
    asm volatile("red.relaxed.cluster.shared::cluster.add.u32 [%0], 1;" ::"r"(addr) : "memory");
}
__device__ __forceinline__ uint32_t cluster_take(uint32_t addr) {
    uint32_t r;
    asm volatile("atom.relaxed.cluster.shared::cluster.add.u32 %0, [%1], 1;" : "=r"(r) : "r"(addr) : "memory");
    return r;
}
__device__ __forceinline__ uint32_t cluster_read(uint32_t addr) {
    uint32_t r;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(r) : "r"(addr) : "memory");
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Counting sort of the samples of one map (MSDA: a batch entry, head and level) by cell, with the counters in the shared
// memory of a cluster of CTAs: atomics there are faster than in L2 (a version with one L2 counter
// per cell took 72 + 42 us at the encoder shape, bound by the rate of L2 atomics). The CTAs of a
// cluster share the samples and the cells of a map: each counts and places its samples,
// whoever holds the counter. Where cells hold many samples each CTA keeps to itself:
// it sorts its own queries (whose runs are then that much shorter). The CTAs' results follow
// each other in the order in which they get there.
template <typename Source>
__global__ void __launch_bounds__(kSortThreads, 2)
sort_cells_kernel(const __grid_constant__ Source src, const __grid_constant__ SortParams sp) {
    extern __shared__ uint32_t s_count[];   // [kSortCells]
    __shared__ uint32_t warp_sum[32];
    __shared__ uint32_t block_sum;           // samples this CTA's counters hold
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (blockIdx.x == 0 && tid == 0) *sp.ticket = 0u;
    if (!src.ok()) {         // the same answer in every CTA
        if (tid == 0) sp.regions[blockIdx.x / sp.parts] = make_uint2(0u, 0u);
        return;
    }

    const uint32_t part = blockIdx.x % sp.parts;   // rank in the cluster
    const typename Source::Map map = src.map(blockIdx.x / sp.parts);
    const uint32_t cells = map.cells, samples = src.samples;
    // on its own: at least sixteen samples per cell are left to each CTA, and the counters fit
    const bool alone = sp.parts == 1 || (samples / sp.parts >= 16u * cells && cells <= kSortCells);
    const uint32_t begin_sample = static_cast<uint32_t>(static_cast<uint64_t>(samples) * part / sp.parts);
    const uint32_t n =
        static_cast<uint32_t>(static_cast<uint64_t>(samples) * (part + 1) / sp.parts) - begin_sample;

    // cells held by one CTA at a time, by all of the cluster (or by this CTA alone) in a pass
    const uint32_t holders = alone ? 1u : sp.parts;
    const uint32_t held = min(kSortCells, (cells + holders - 1) / holders);
    const uint32_t pass_cells = held * holders;
    const FastDiv by_held = sp.parts == 1 ? FastDiv{0u, 0u} : device_fastdiv(held);
    auto sync = [&]() {
        if (alone) __syncthreads();
        else cluster_barrier();
    };
    const uint32_t region = (blockIdx.x / sp.parts) * samples;
    uint32_t placed = 0;         // samples of the region placed by earlier passes
    constexpr uint32_t kU = 4;   // samples in flight per thread
    for (uint32_t lo = 0; lo < cells; lo += pass_cells) {
        for (uint32_t i = tid; i < held; i += kSortThreads) s_count[i] = 0u;
        sync();
        for (uint32_t i0 = tid; i0 < n; i0 += kU * kSortThreads) {
            float2 xy[kU];
            uint32_t id[kU];
#pragma unroll
            for (uint32_t u = 0; u < kU; ++u) {
                const uint32_t i = i0 + u * kSortThreads;
                id[u] = src.id(map, begin_sample + (i < n ? i : 0u));
                xy[u] = src.position(id[u]);
            }
#pragma unroll
            for (uint32_t u = 0; u < kU; ++u) {
                if (i0 + u * kSortThreads >= n) break;
                const uint32_t c = src.cell(map, xy[u]);
                if (c - lo < pass_cells) {
                    if (alone) {
                        atomicAdd(s_count + (c - lo), 1u);
                    } else {
                        const uint32_t rank = fd_div(c - lo, by_held);
                        cluster_count(cluster_address(s_count + (c - lo - rank * held), rank));
                    }
                } else if (c == kNoRow && lo == 0) {
                    src.drop(id[u]);
                }
            }
        }
        sync();
        // counts -> first positions: a thread takes an odd number of neighbours (no bank conflicts)
        const uint32_t per = ((held + kSortThreads - 1) / kSortThreads) | 1u;
        const uint32_t begin = min(held, tid * per), stop = min(held, begin + per);
        uint32_t sum = 0;
        for (uint32_t i = begin; i < stop; ++i) sum += s_count[i];
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) warp_sum[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            const uint32_t mine = warp_sum[lane];
            uint32_t w = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += v;
            }
            warp_sum[lane] = w - mine;
            if (lane == 31) block_sum = w;
        }
        if (sp.parts == 1) __syncthreads();
        else cluster_barrier();
        // the samples of lower ranks come first
        uint32_t at = region + placed + warp_sum[warp] + incl - sum;
        for (uint32_t r = 0; r < sp.parts; ++r) {
            const uint32_t m = sp.parts == 1 ? block_sum : cluster_read(cluster_address(&block_sum, r));
            if (r < part) at += m;
            placed += m;
        }
        for (uint32_t i = begin; i < stop; ++i) {
            const uint32_t m = s_count[i];
            s_count[i] = at;
            at += m;
        }
        sync();
        for (uint32_t i0 = tid; i0 < n; i0 += kU * kSortThreads) {
            float2 xy[kU];
            uint32_t id[kU], pos[kU];
#pragma unroll
            for (uint32_t u = 0; u < kU; ++u) {
                const uint32_t i = i0 + u * kSortThreads;
                id[u] = src.id(map, begin_sample + (i < n ? i : 0u));
                xy[u] = src.position(id[u]);
                pos[u] = kNoRow;
            }
#pragma unroll
            for (uint32_t u = 0; u < kU; ++u) {
                if (i0 + u * kSortThreads >= n) break;
                const uint32_t c = src.cell(map, xy[u]);
                if (c - lo < pass_cells) {
                    if (alone) {
                        pos[u] = atomicAdd(s_count + (c - lo), 1u);
                    } else {
                        const uint32_t rank = fd_div(c - lo, by_held);
                        pos[u] = cluster_take(cluster_address(s_count + (c - lo - rank * held), rank));
                    }
                }
            }
#pragma unroll
            for (uint32_t u = 0; u < kU; ++u)
                if (pos[u] != kNoRow) sp.sorted[pos[u]] = id[u];
        }
        // nobody leaves, or clears the counters, while others still use them
        if (sp.parts == 1) __syncthreads();
        else cluster_barrier();
    }
    if (tid == 0 && part == 0) sp.regions[blockIdx.x / sp.parts] = make_uint2(region, placed);
}

// Warps draw tickets in order; a ticket is up to `len` consecutive sorted samples of one region.
struct Ticket {
    uint32_t begin, end;   // positions; begin >= end: nothing
};
__device__ __forceinline__ bool next_ticket(const SortParams& sp, uint32_t len, int lane, Ticket& t) {
    uint32_t n = 0;
    if (lane == 0) n = atomicAdd(sp.ticket, 1u);
    n = __shfl_sync(0xffffffffu, n, 0);
    if (n >= sp.tickets) return false;
    const uint32_t region = fd_div(n, sp.fd_tickets);
    const uint2 r = __ldg(sp.regions + region);
    t.begin = r.x + (n - region * sp.tickets_per_region) * len;
    t.end = min(r.x + r.y, t.begin + len);
    return true;
}

// Four channels of a row, as two fp32 pairs.
template <typename T>
__device__ __forceinline__ void load_quad(const T* p, f32x2 (&q)[2]) {
    if constexpr (sizeof(T) == 4) {
        const ulonglong2 r = __ldg(reinterpret_cast<const ulonglong2*>(p));
        q[0] = r.x;
        q[1] = r.y;
    } else {
        const uint2 r = __ldg(reinterpret_cast<const uint2*>(p));
        const uint32_t w[2] = {r.x, r.y};
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if constexpr (std::is_same<T, __half>::value) {
                const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
                q[i] = pack2(v.x, v.y);
            } else {
                q[i] = pack2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
            }
        }
    }
}
__device__ __forceinline__ void red_quad(float* p, const f32x2 (&q)[2]) {
    const float2 a = unpack2(q[0]), b = unpack2(q[1]);
    red_add_f32x4(p, a.x, a.y, b.x, b.y);
}

// Sums each of N per-lane values over groups of LPR lanes (N a power of two <= LPR): halving
// steps in which a lane gives half of its values away and keeps the other half, then plain
// steps. Lane j of a group ends up with the sum of value j / (LPR / N).
template <int N, int LPR, typename V>
__device__ __forceinline__ V reduce_values(V (&d)[N], int j) {
    if constexpr (N == 1) {
#pragma unroll
        for (int o = LPR / 2; o >= 1; o >>= 1) d[0] += __shfl_xor_sync(0xffffffffu, d[0], o);
        return d[0];
    } else {
        const bool up = (j & (LPR / 2)) != 0;
        V half[N / 2];
#pragma unroll
        for (int i = 0; i < N / 2; ++i) {
            half[i] = up ? d[N / 2 + i] : d[i];
            half[i] += __shfl_xor_sync(0xffffffffu, up ? d[i] : d[N / 2 + i], LPR / 2);
        }
        return reduce_values<N / 2, LPR / 2>(half, j);
    }
}

// Tickets and grid of a main kernel with `streams` per warp, a round of 32 samples being
// 32 / streams steps of each.
static cudaError_t plan_tickets(const void* kernel, int streams, SortParams& sp,
                                uint32_t samples_per_map, const LaunchShape& ls, uint32_t* grid) {
    int per_sm = ls.ctas_per_sm;
    if (per_sm <= 0) {
        const cudaError_t e = resident_ctas(kernel, kThreadsPerCta, 0, &per_sm);
        if (e != cudaSuccess) return e;
    }
    const uint32_t cap = static_cast<uint32_t>(ls.sm_count) * per_sm;
    // Long streams enter fewer cells, short ones level the load: eight tickets per resident
    // warp, as long as a stream keeps one round.
    const uint32_t want = sp.nsamples / (cap * kWarpsPerCta * 8u * streams);
    const uint32_t round = 32u / streams;
    sp.stream = want / round * round;
    if (sp.stream < round) sp.stream = round;
    if (sp.stream > kMaxStream) sp.stream = kMaxStream;
    const uint32_t len = sp.stream * streams;
    sp.tickets_per_region = (samples_per_map + len - 1) / len;
    sp.fd_tickets = make_fastdiv(sp.tickets_per_region);
    sp.tickets = sp.nregions * sp.tickets_per_region;
    const uint32_t need = (sp.tickets + kWarpsPerCta - 1) / kWarpsPerCta;
    *grid = need < cap ? need : cap;
    return cudaSuccess;
}

template <typename Source>
static cudaError_t launch_sort(const Source& src, uint32_t maps, SortParams& sp, int sm_count,
                               cudaStream_t stream) {
    auto kern = sort_cells_kernel<Source>;
    const size_t smem = kSortCells * sizeof(uint32_t);
    int resident = 0;   // (asked for the shared-memory limit that the call sets)
    const cudaError_t e = resident_ctas(reinterpret_cast<const void*>(kern), kSortThreads, smem, &resident);
    if (e != cudaSuccess) return e;
    // the smallest cluster that gives most SMs work
    sp.parts = 1;
    while (sp.parts < kMaxSortParts && maps * sp.parts < 3u * sm_count / 2u) sp.parts *= 2;
    sp.nregions = maps;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(maps * sp.parts);
    cfg.blockDim = dim3(kSortThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = sp.parts;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, src, sp);
}

}  // namespace msda
