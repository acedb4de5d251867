// Counting sort of samples by the cell of the map they fall into, and what the kernels that walk
// the sorted samples share: the backward of the attention operators (msda_bwd_sorted.cuh) and of
// deformable aggregation (da_sorted_sm100.cu).
#pragma once

#include <algorithm>
#include <type_traits>

#include "msda_common.cuh"
#include "msda_launch.h"
#include "sort_plan.h"

namespace msda {

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

// Zeros for `bytes` bytes from p on, by thread `first` of `step`.
__device__ __forceinline__ void clear_bytes(void* p, size_t bytes, size_t first, size_t step) {
    unsigned char* at = static_cast<unsigned char*>(p);
    const size_t head = min(bytes, static_cast<size_t>((16u - (reinterpret_cast<uintptr_t>(at) & 15u)) & 15u));
    uint4* body = reinterpret_cast<uint4*>(at + head);
    const size_t pieces = (bytes - head) / 16, tail = head + pieces * 16;
    for (size_t i = first; i < pieces; i += step) body[i] = make_uint4(0u, 0u, 0u, 0u);
    if (first < head) at[first] = 0;
    if (first < bytes - tail) at[tail + first] = 0;
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
__device__ __forceinline__ void cluster_write(uint32_t addr, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Counting sort of the samples of one map (MSDA: a batch entry, head and level) by cell, by a cluster of
// CTAs that share the map's samples, with the counters in their shared memory (one L2 counter per cell:
// 114 us at the encoder shape). Bound by scattered accesses of 4 bytes: one store per sample in any
// case, some 200 G per second through L2, and what passes between the CTAs of a cluster, a few bytes per
// clock and SM. So the counters are kept in one of three ways, by samples per cell:
//   split   every CTA holds a part of the cells, all count and place in them with remote atomics: two
//           remote accesses per sample;
//   merged  every CTA counts its samples on its own, then the CTAs turn a slice of the cells each into
//           first positions for all (cell by cell, a cell's parts by CTA): three remote accesses, side
//           by side, per cell and CTA;
//   alone   many samples per cell: every CTA sorts its samples on its own, the results follow each other.

// One CTA's part of the sort of a map; returns how many of the map's samples have a place.
template <Counters KEPT, typename Source>
__device__ __forceinline__ uint32_t sort_map(const Source& src, const SortParams& sp,
                                             const typename Source::Map& map, uint32_t* s_count,
                                             uint32_t* warp_sum, uint32_t* block_sum) {
    constexpr bool kSplit = KEPT == Counters::kSplit, kMerged = KEPT == Counters::kMerged;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t parts = sp.parts, part = blockIdx.x % parts;   // rank in the cluster
    const uint32_t samples = src.samples, cells = map.cells;
    const uint32_t begin_sample = static_cast<uint32_t>(static_cast<uint64_t>(samples) * part / parts);
    const uint32_t n =
        static_cast<uint32_t>(static_cast<uint64_t>(samples) * (part + 1) / parts) - begin_sample;
    auto sync = [&]() {
        if (!kSplit && !kMerged) __syncthreads();
        else cluster_barrier();
    };

    // A thread's samples are a whole number of periods apart (a period: the points of a query), which
    // makes their numbers an arithmetic sequence: no division per sample.
    const uint32_t periods = kSortThreads / src.period, threads = periods * src.period;
    const uint32_t first = tid < threads ? tid : n, id_step = periods * src.period_step;
    const uint32_t first_id = src.id(map, begin_sample + (first < n ? first : 0u));

    // cells held by a CTA at a time, and by all of the cluster in a pass
    const uint32_t held = min(kSortCells, kSplit ? (cells + parts - 1) / parts : cells);
    const uint32_t pass_cells = kSplit ? held * parts : held;
    const FastDiv by_held = kSplit ? device_fastdiv(held) : FastDiv{0u, 0u};
    auto remote = [&](uint32_t c) {   // the counter of cell c of the pass
        const uint32_t rank = fd_div(c, by_held);
        return cluster_address(s_count + (c - rank * held), rank);
    };

    // room for the sorted numbers, which then leave side by side (96 maps of 107 K samples on 375 cells:
    // 97 us before, 81 now)
    const bool staged = KEPT == Counters::kAlone && cells + n <= sp.room;
    uint32_t placed = 0;         // samples of the map placed by earlier passes
    constexpr uint32_t kU = Source::kInFlight;   // samples in flight per thread
    // each(cell of this pass, sample number)
    auto for_each_sample = [&](uint32_t lo, auto&& each) {
        uint32_t id = first_id;
        for (uint32_t i0 = first; i0 < n; i0 += kU * threads) {
            float2 xy[kU];
#pragma unroll
            for (uint32_t u = 0; u < kU; ++u)
                xy[u] = src.position(i0 + u * threads < n ? id + u * id_step : first_id);
#pragma unroll
            for (uint32_t u = 0; u < kU; ++u) {
                if (i0 + u * threads >= n) break;
                const uint32_t c = src.cell(map, xy[u]) - lo;   // (none: far beyond the pass)
                if (c < pass_cells) each(c, id + u * id_step);
            }
            id += kU * id_step;
        }
    };
    for (uint32_t lo = 0; lo < cells; lo += pass_cells) {
        for (uint32_t i = tid; i < held; i += kSortThreads) s_count[i] = 0u;
        sync();
        for_each_sample(lo, [&](uint32_t c, uint32_t) {
            if (kSplit) cluster_count(remote(c));
            else atomicAdd(s_count + c, 1u);
        });
        sync();
        // counts -> first positions: of this CTA's counters, or, merged, of a slice of everybody's. A
        // warp takes a range of whole groups of 32 cells.
        const uint32_t slice = kMerged ? (held + parts - 1) / parts : held;
        const uint32_t slice_begin = kMerged ? part * slice : 0u, slice_end = min(held, slice_begin + slice);
        const uint32_t range = ((slice + kSortThreads - 1) / kSortThreads) * 32u;
        const uint32_t begin = slice_begin + warp * range, stop = min(slice_end, begin + range);
        // a cell's counts; a CTA begins with its own counter and goes on to another one than the others
        uint32_t m[kMaxSortParts];
        auto count_of = [&](uint32_t i) {
            uint32_t all = m[0] = s_count[i];
            if (kMerged) {
#pragma unroll
                for (uint32_t r = 1; r < kMaxSortParts; ++r)
                    m[r] = r < parts ? cluster_read(cluster_address(s_count + i, r ^ part)) : 0u;
#pragma unroll
                for (uint32_t r = 1; r < kMaxSortParts; ++r) all += m[r];
            }
            return all;
        };
        uint32_t sum = 0;
        for (uint32_t i = begin + lane; i < stop; i += 32) sum += count_of(i);
        sum = __reduce_add_sync(0xffffffffu, sum);
        if (lane == 0) warp_sum[warp] = sum;
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
            if (lane == 31) *block_sum = w;
        }
        if (parts == 1) __syncthreads();
        else cluster_barrier();
        // what lower ranks hold comes first
        uint32_t base = blockIdx.x / parts * samples + placed;
        for (uint32_t r = 0; r < parts; ++r) {
            const uint32_t there = parts == 1 ? *block_sum : cluster_read(cluster_address(block_sum, r));
            if (r < part) base += there;
            placed += there;
        }
        uint32_t at = warp_sum[warp] + (staged ? 0u : base);
        for (uint32_t i0 = begin; i0 < stop; i0 += 32) {
            const uint32_t i = i0 + lane;
            const uint32_t count = i < stop ? count_of(i) : 0u;
            uint32_t incl = count;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            if (i < stop) {
                uint32_t pos = at + incl - count;
                s_count[i] = pos;
                if (kMerged) {
#pragma unroll
                    for (uint32_t r = 1; r < kMaxSortParts; ++r) {
                        pos += m[r - 1];
                        if (r < parts) cluster_write(cluster_address(s_count + i, r ^ part), pos);
                    }
                }
            }
            at += __shfl_sync(0xffffffffu, incl, 31);
        }
        sync();
        if (!staged) {
            for_each_sample(lo, [&](uint32_t c, uint32_t id) {
                sp.sorted[kSplit ? cluster_take(remote(c)) : atomicAdd(s_count + c, 1u)] = id;
            });
        } else {
            uint32_t* to = s_count + held;
            for_each_sample(lo, [&](uint32_t c, uint32_t id) { to[atomicAdd(s_count + c, 1u)] = id; });
            __syncthreads();
            for (uint32_t i = tid; i < *block_sum; i += kSortThreads) sp.sorted[base + i] = to[i];
        }
        // nobody leaves, or clears the counters, while others still use them
        if (parts == 1) __syncthreads();
        else cluster_barrier();
    }
    return placed;
}

// KEPT: the one way, for maps that are all alike (a kernel that holds all three spills more; 18 and 12
// convolution maps of 13 K samples: 26.6 and 26.0 us, now 13.7 and 10.0); -1: chosen map by map.
template <typename Source, int KEPT>
__global__ void __launch_bounds__(kSortThreads, 2)
sort_cells_kernel(const __grid_constant__ Source src, const __grid_constant__ SortParams sp) {
    extern __shared__ uint32_t s_count[];   // [sp.room]: counters, then staged sample numbers
    __shared__ uint32_t warp_sum[32];
    __shared__ uint32_t block_sum;           // samples this CTA's counters, or slice of them, hold
    // CTAs past those that sort (whole clusters) fill with zeros what the main kernel adds to or may
    // leave out: the sort leaves most of the memory's rate to them
    const uint32_t sorting = sp.nregions * sp.parts;
    if (blockIdx.x >= sorting) {
        const size_t first = static_cast<size_t>(blockIdx.x - sorting) * kSortThreads + threadIdx.x;
        const size_t step = static_cast<size_t>(gridDim.x - sorting) * kSortThreads;
        if (sp.clear_sums) clear_bytes(src.sums(), src.sums_bytes(), first, step);
        src.clear(first, step);
        return;
    }
    if (gridDim.x == sorting)   // no room beside them
        src.clear(static_cast<size_t>(blockIdx.x) * kSortThreads + threadIdx.x,
                  static_cast<size_t>(sorting) * kSortThreads);
    if (blockIdx.x == 0 && threadIdx.x == 0) *sp.ticket = 0u;
    const uint32_t parts = sp.parts, region = blockIdx.x / parts;
    if (!src.ok()) {         // the same answer in every CTA
        if (threadIdx.x == 0) sp.regions[region] = make_uint2(0u, 0u);
        return;
    }
    const typename Source::Map map = src.map(region);
    const Counters kept = KEPT >= 0 ? static_cast<Counters>(KEPT) : counters_of(parts, src.samples, map.cells);
    uint32_t placed;
    if (kept == Counters::kAlone)
        placed = sort_map<Counters::kAlone>(src, sp, map, s_count, warp_sum, &block_sum);
    else if (kept == Counters::kMerged)
        placed = sort_map<Counters::kMerged>(src, sp, map, s_count, warp_sum, &block_sum);
    else
        placed = sort_map<Counters::kSplit>(src, sp, map, s_count, warp_sum, &block_sum);
    if (threadIdx.x == 0 && blockIdx.x % parts == 0) sp.regions[region] = make_uint2(region * src.samples, placed);
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
    // Long streams enter fewer cells, short ones level the load: eight tickets per resident warp, or as
    // few as two where a stream would be under 32 samples (2.6 M samples, 4 per cell, 4 streams:
    // 217 us with 16 samples per stream, 194 with 32; 1.3 M at 2.6 per cell 178 with 8, 120 with 32).
    const uint32_t warps = cap * kWarpsPerCta * streams, round = 32u / streams;
    const uint32_t want = std::max(sp.nsamples / (warps * 8u), std::min(32u, sp.nsamples / (warps * 2u)));
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
    const SortChoice choice = choose_sort({maps, src.samples, src.mean_cells, src.most_cells},
                                          static_cast<uint32_t>(sm_count), Source::kMapsAlike);
    sp.parts = choice.parts;
    sp.room = choice.room;
    sp.nregions = maps;
    void (*kern)(const Source, const SortParams) = nullptr;
    if constexpr (Source::kMapsAlike) {
        const Counters kept = counters_of(sp.parts, src.samples, src.most_cells);
        kern = kept == Counters::kAlone    ? sort_cells_kernel<Source, static_cast<int>(Counters::kAlone)>
               : kept == Counters::kMerged ? sort_cells_kernel<Source, static_cast<int>(Counters::kMerged)>
                                           : sort_cells_kernel<Source, static_cast<int>(Counters::kSplit)>;
    } else {
        kern = sort_cells_kernel<Source, -1>;
    }
    const size_t smem = sp.room * sizeof(uint32_t);
    int resident = 0;   // (asked for the shared-memory limit that the call sets)
    const cudaError_t e = resident_ctas(reinterpret_cast<const void*>(kern), kSortThreads, smem, &resident);
    if (e != cudaSuccess) return e;
    // The sums are filled with zeros beside the sort where that leaves CTAs room and takes about as
    // long (192 maps of 20 K samples, 189 MB: 51 + 32 -> 61 us; 16 of 160 K, 82 MB: 59 + 15 -> 60), and
    // by a memset otherwise (256 of 80 K, 490 MB: 194 + 79 -> 314; key points, 553 MB: 17 + 104 -> 123).
    const bool room = maps * sp.parts <= 3u * sm_count / 2u;
    const bool beside = room && src.sums_bytes() / 6e3 <= 1.5 * choice.ns;
    sp.clear_sums = beside ? 1u : 0u;
    if (!beside && src.sums_bytes() > 0) {
        const cudaError_t err = cudaMemsetAsync(src.sums(), 0, src.sums_bytes(), stream);
        if (err != cudaSuccess) return err;
    }
    // the zeros: 128 KB or more for a CTA, whole clusters, at most two CTAs per SM (those that find no room
    // beside the sorting ones follow them); where that is too few the sorting CTAs see to them first (256
    // maps of 80 K: 194 us against 209 after the others)
    size_t clearing = ((beside ? src.sums_bytes() : 0) + src.clear_size() + (128u << 10) - 1) >> 17;
    if (!room) clearing = 0;
    clearing = std::min<size_t>(clearing, 2u * sm_count);
    clearing = (clearing + sp.parts - 1) / sp.parts * sp.parts;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(maps * sp.parts + clearing));
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
