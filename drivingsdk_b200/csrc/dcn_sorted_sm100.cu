// The sampling halves of the deformable convolution over cell-sorted samples (cell_sort.cuh), for
// sm_100a. A sample is a (pixel, deformable group, tap) with the Cd channels of its group; it meets the
// four corner rows V_c of x around its position with bilinear weights b_c:
//   forward    its row of the columns = mask * sum_c b_c V_c, written as fp16 pairs
//   backward   with its row g of grad_columns and t_c = <V_c, g>:  grad_x[V_c] += mask * b_c * g,
//              grad_mask = sum_c b_c t_c, grad_offset = mask * (differences of the t_c)
// Taken pixel by pixel (gather_pairs_kernel, dcn_sample_kernel) every sample loads four rows, 1.9 GB
// at the operator's test shape, and reduces as many: 168 and 385 us, bound by the return path of
// 128-bit loads and by the reductions. With a 3 x 3 kernel some nine samples share a cell: sorted
// by cell, corner rows and their sums stay in registers and what is left is to write or read the
// columns once (481 MB): 98 and 159 us, plus 14 us for the sort, which both directions use.
// One sample at a time per warp, lane = channel quads j and j + 32 of a slice of NV * 128 channels;
// backward slices add their parts of the t_c up with atomics.
#include "cell_sort.cuh"
#include "dcn_common.cuh"
#include "dcn_split.h"
#include "split_scale.cuh"

namespace dcn {
namespace {

using namespace msda;

// What the sort needs to know: a map is one (image, deformable group).
struct ConvSamples {
    // Samples in flight per thread of the sort: a position takes two loads and five divisions, so more
    // than one spills (18 maps of 13 K samples, alone: 15.5 us with one, 19.6 with two, 26 with four).
    static constexpr uint32_t kInFlight = 1;
    static constexpr bool kMapsAlike = true;    // all have the same cells
    DcnParams p;
    uint32_t samples;   // of one map: Ho * Wo * K
    uint32_t period, period_step;   // K, DG * K
    uint32_t most_cells, mean_cells;   // of a map

    struct Map {
        uint32_t cells, n, dg;
    };
    __device__ __forceinline__ bool ok() const { return true; }
    __device__ __forceinline__ Map map(uint32_t m) const {
        Map r;
        // the last one takes the samples outside the image, whose columns and gradients are zero
        r.cells = static_cast<uint32_t>(p.H + 1) * static_cast<uint32_t>(p.W + 1) + 1u;
        r.n = m / p.DG;
        r.dg = m - r.n * p.DG;
        return r;
    }
    __device__ __forceinline__ uint32_t id(const Map& m, uint32_t i) const {
        const uint32_t pixel = fd_div(i, p.fd_K);
        return ((m.n * p.HoWo + pixel) * p.DG + m.dg) * p.K + (i - pixel * p.K);
    }
    __device__ __forceinline__ float2 position(uint32_t id) const { return sample_position(p, id).at; }
    __device__ __forceinline__ uint32_t cell(const Map& m, float2 at) const {
        if (!inside(p, at)) return m.cells - 1u;
        return static_cast<uint32_t>(__float2int_rd(at.x) + 1) * static_cast<uint32_t>(p.W + 1) +
               static_cast<uint32_t>(__float2int_rd(at.y) + 1);
    }
    // nothing to clear: every sample has a cell, and the caller clears the gradients
    __host__ __device__ void* sums() const { return nullptr; }
    __host__ __device__ size_t sums_bytes() const { return 0; }
    size_t clear_size() const { return 0; }
    __device__ __forceinline__ void clear(size_t, size_t) const {}
    static __device__ __forceinline__ bool inside(const DcnParams& p, float2 at) {   // false for NaN
        return at.x > -1.f && at.y > -1.f && at.x < static_cast<float>(p.H) && at.y < static_cast<float>(p.W);
    }

    struct Position {
        float2 at;          // (y, x)
        uint32_t m, dg, k;
    };
    static __device__ __forceinline__ Position sample_position(const DcnParams& p, uint32_t id) {
        Position r;
        const uint32_t t = fd_div(id, p.fd_K);
        r.k = id - t * p.K;
        r.m = fd_div(t, p.fd_DG);
        r.dg = t - r.m * p.DG;
        const uint32_t n = fd_div(r.m, p.fd_HoWo);
        const uint32_t pixel = r.m - n * p.HoWo;
        const uint32_t ho = fd_div(pixel, p.fd_Wo), wo = pixel - ho * p.Wo;
        const uint32_t ki = fd_div(r.k, p.fd_kw), kj = r.k - ki * p.kw;
        const float2 d = __ldg(reinterpret_cast<const float2*>(p.offset) + id);
        r.at.x = static_cast<float>(static_cast<int>(ho) * p.sh - p.ph + static_cast<int>(ki) * p.dh) + d.x;
        r.at.y = static_cast<float>(static_cast<int>(wo) * p.sw - p.pw + static_cast<int>(kj) * p.dw) + d.y;
        return r;
    }
};

// Tickets of the slices of one run follow each other.
__device__ __forceinline__ bool next_slice_ticket(const SortParams& sp, uint32_t slices, int lane, Ticket& t,
                                                  uint32_t& region, uint32_t& slice) {
    uint32_t n = 0;
    if (lane == 0) n = atomicAdd(sp.ticket, 1u);
    n = __shfl_sync(0xffffffffu, n, 0);
    const uint32_t run = n / slices;
    slice = n - run * slices;
    if (run >= sp.tickets) return false;
    region = fd_div(run, sp.fd_tickets);
    const uint2 r = __ldg(sp.regions + region);
    t.begin = r.x + (run - region * sp.tickets_per_region) * sp.stream;
    t.end = min(r.x + r.y, t.begin + sp.stream);
    return true;
}

// A sorted sample, set up by its lane.
struct Record {
    ulonglong2 w01, w23;             // mask * bilinear weights, each twice (packed multiply-add)
    float lh, lw, mask;
    uint32_t id, columns, row, cell, pad;   // offsets in quads; cell: existing corners
};
__device__ __forceinline__ Record set_up_record(const DcnParams& p, const SortParams& sp, uint32_t at,
                                                bool live, uint32_t n_image, uint32_t units) {
    Record r;
    r.id = r.columns = r.row = r.cell = r.pad = 0u;
    r.lh = r.lw = r.mask = 0.f;
    r.w01 = r.w23 = make_ulonglong2(0ull, 0ull);
    if (!live) return r;
    r.id = __ldg(sp.sorted + at);
    const ConvSamples::Position s = ConvSamples::sample_position(p, r.id);
    r.columns = s.m * (static_cast<uint32_t>(p.G) * p.K * (p.Cg / 4)) + s.k * (p.Cg / 4);
    if (!ConvSamples::inside(p, s.at)) return r;   // no corner
    r.mask = p.mask != nullptr ? __ldg(p.mask + r.id) : 1.f;
    const float y0f = floorf(s.at.x), x0f = floorf(s.at.y);
    const int y0 = static_cast<int>(y0f), x0 = static_cast<int>(x0f);
    r.lh = s.at.x - y0f;
    r.lw = s.at.y - x0f;
    const float hh = 1.f - r.lh, hw = 1.f - r.lw;
    const uint32_t sides = (x0 >= 0 ? 1u : 0u) | (x0 + 1 < p.W ? 2u : 0u);
    r.cell = (y0 >= 0 ? sides : 0u) | (y0 + 1 < p.H ? sides << 2 : 0u);
    r.row = (n_image * static_cast<uint32_t>(p.H * p.W) + static_cast<uint32_t>(y0 * p.W + x0)) * units;
    const float a = hh * hw * r.mask, b = hh * r.lw * r.mask;
    const float c = r.lh * hw * r.mask, d = r.lh * r.lw * r.mask;
    r.w01 = make_ulonglong2(pack2(a, a), pack2(b, b));
    r.w23 = make_ulonglong2(pack2(c, c), pack2(d, d));
    return r;
}

// What a lane keeps for a ticket: its quads, and where they lie in the columns of a (pixel, tap).
template <int NV>
struct LaneSlice {
    bool on[NV];
    uint32_t column_at[NV];
    size_t x_at;          // floats
    __device__ __forceinline__ LaneSlice(const DcnParams& p, uint32_t dg, uint32_t slice, int lane) {
        const int first = static_cast<int>(slice) * (NV * 32) + lane;
        x_at = static_cast<size_t>(dg) * p.Cd + first * 4;
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            const int quad = first + 32 * k;
            on[k] = quad * 4 < p.Cd;
            const uint32_t c = dg * p.Cd + (on[k] ? quad * 4 : 0);
            const uint32_t g = fd_div(c, p.fd_Cg);
            column_at[k] = (g * p.K * p.Cg + (c - g * p.Cg)) / 4;
        }
    }
};

// Forward. The bound of the columns gives the scale of the pairs, their range the form.
template <int NV>
__global__ void __launch_bounds__(kThreadsPerCta, NV > 1 ? 3 : 4)
gather_sorted_kernel(const __grid_constant__ DcnParams p, const __grid_constant__ SortParams sp,
                     uint32_t slices, const __grid_constant__ ColumnsOut out) {
    __shared__ __align__(16) Record s_rec[kWarpsPerCta][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t units = static_cast<uint32_t>(p.C) / 4, step_y = static_cast<uint32_t>(p.W) * units;
    const float scale = exp2_int(split_exponent(out.bound, 0));
    const bool pairs = !range_is_wide(out.range), plain = !pairs || out.keep_f32;

    Ticket ticket;
    uint32_t region, slice;
    while (next_slice_ticket(sp, slices, lane, ticket, region, slice)) {
        if (ticket.begin >= ticket.end) continue;
        const uint32_t n_image = region / p.DG, dg = region - n_image * p.DG;
        const LaneSlice<NV> ls(p, dg, slice, lane);
        const float* x = p.x + ls.x_at;
        f32x2 val[4][NV][2];
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int k = 0; k < NV; ++k) val[c][k][0] = val[c][k][1] = 0ull;
        uint32_t cur = 0u, cell = 0u;
        auto fetch = [&](int c) {
            const size_t off =
                static_cast<size_t>(cur + ((c & 1) ? units : 0u) + ((c & 2) ? step_y : 0u)) * 4;
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                val[c][k][0] = val[c][k][1] = 0ull;
                if (((cell >> c) & 1u) && ls.on[k]) load_quad<float>(x + off + k * 128, val[c][k]);
            }
        };
        for (uint32_t at = ticket.begin; at < ticket.end; at += 32) {
            const int n = min(32, static_cast<int>(ticket.end - at));
            const Record r = set_up_record(p, sp, at + lane, lane < n, n_image, units);
            uint32_t prow = __shfl_up_sync(0xffffffffu, r.row, 1);
            uint32_t pcell = __shfl_up_sync(0xffffffffu, r.cell, 1);
            if (lane == 0) {
                prow = cur;
                pcell = cell;
            }
            const uint32_t m_enter =
                __ballot_sync(0xffffffffu, lane < n && (r.row != prow || r.cell != pcell));
            const uint32_t m_right = __ballot_sync(
                0xffffffffu, r.row == prow + units && ((pcell >> 1) & 5u) == (r.cell & 5u));
            s_rec[warp][lane] = r;
            __syncwarp();
#pragma unroll 1
            for (int i = 0; i < n; ++i) {
                const Record& q = s_rec[warp][i];
                if ((m_enter >> i) & 1u) {
                    cur = q.row;
                    cell = q.cell;
                    if ((m_right >> i) & 1u) {
#pragma unroll
                        for (int c = 0; c < 4; c += 2)
#pragma unroll
                            for (int k = 0; k < NV; ++k) {
                                val[c][k][0] = val[c + 1][k][0];
                                val[c][k][1] = val[c + 1][k][1];
                            }
                    } else {
                        fetch(0);
                        fetch(2);
                    }
                    fetch(1);
                    fetch(3);
                }
                const f32x2 w[4] = {q.w01.x, q.w01.y, q.w23.x, q.w23.y};
#pragma unroll
                for (int k = 0; k < NV; ++k) {
                    uint2 part[2];
                    float2 v[2];
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        f32x2 sum = mul2(w[0], val[0][k][e]);
#pragma unroll
                        for (int c = 1; c < 4; ++c) sum = fma2(w[c], val[c][k][e], sum);
                        v[e] = unpack2(sum);
                        part[e] = split_pair(v[e].x, v[e].y, scale);
                    }
                    if (ls.on[k]) {
                        const size_t to_at = (static_cast<size_t>(q.columns) + ls.column_at[k]) * 4;
                        if (pairs) {
                            uint16_t* to = out.pairs + to_at;
                            *reinterpret_cast<uint2*>(to) = make_uint2(part[0].x, part[1].x);
                            *reinterpret_cast<uint2*>(to + out.plane) = make_uint2(part[0].y, part[1].y);
                        }
                        if (plain)
                            *reinterpret_cast<float4*>(out.f32 + to_at) =
                                make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
                    }
                }
            }
            __syncwarp();
        }
    }
}

template <int NV>
__global__ void __launch_bounds__(kThreadsPerCta, NV > 1 ? 2 : 3)
scatter_sorted_kernel(const __grid_constant__ DcnParams p, const __grid_constant__ SortParams sp,
                      uint32_t slices) {
    constexpr int U = 4;    // samples in flight (512 channels: 180 us with two, 159 with four, though 52 bytes spill)
    __shared__ __align__(16) Record s_rec[kWarpsPerCta][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t units = static_cast<uint32_t>(p.C) / 4, step_y = static_cast<uint32_t>(p.W) * units;

    Ticket ticket;
    uint32_t region, slice;
    while (next_slice_ticket(sp, slices, lane, ticket, region, slice)) {
        if (ticket.begin >= ticket.end) continue;
        const uint32_t n_image = region / p.DG, dg = region - n_image * p.DG;
        const LaneSlice<NV> ls(p, dg, slice, lane);
        const float* x = p.x + ls.x_at;
        float* gx = p.grad_x + ls.x_at;

        f32x2 acc[4][NV][2], val[4][NV][2];
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int k = 0; k < NV; ++k) acc[c][k][0] = acc[c][k][1] = val[c][k][0] = val[c][k][1] = 0ull;
        uint32_t cur = 0u, cell = 0u;    // no corner: nothing to flush
        auto offset = [&](int c) {
            return static_cast<size_t>(cur + ((c & 1) ? units : 0u) + ((c & 2) ? step_y : 0u)) * 4;
        };
        auto flush = [&](int c) {
            if ((cell >> c) & 1u) {
#pragma unroll
                for (int k = 0; k < NV; ++k)
                    if (ls.on[k]) red_quad(gx + offset(c) + k * 128, acc[c][k]);
            }
#pragma unroll
            for (int k = 0; k < NV; ++k) acc[c][k][0] = acc[c][k][1] = 0ull;
        };
        auto fetch = [&](int c) {
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                val[c][k][0] = val[c][k][1] = 0ull;
                if (((cell >> c) & 1u) && ls.on[k]) load_quad<float>(x + offset(c) + k * 128, val[c][k]);
            }
        };
        for (uint32_t at = ticket.begin; at < ticket.end; at += 32) {
            // ---- lane = sample: cell, corner weights --------------------------------------
            const int n = min(32, static_cast<int>(ticket.end - at));
            const Record r = set_up_record(p, sp, at + lane, lane < n, n_image, units);
            uint32_t prow = __shfl_up_sync(0xffffffffu, r.row, 1);
            uint32_t pcell = __shfl_up_sync(0xffffffffu, r.cell, 1);
            if (lane == 0) {
                prow = cur;
                pcell = cell;
            }
            const uint32_t m_enter =
                __ballot_sync(0xffffffffu, lane < n && (r.row != prow || r.cell != pcell));
            // one cell to the right: the right corners become the left ones
            const uint32_t m_right = __ballot_sync(
                0xffffffffu, r.row == prow + units && ((pcell >> 1) & 5u) == (r.cell & 5u));
            s_rec[warp][lane] = r;
            __syncwarp();

            // ---- warp = sample --------------------------------------------------------------
#pragma unroll 1
            for (int i0 = 0; i0 < n; i0 += U) {
                f32x2 g[U][NV][2];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint32_t from = s_rec[warp][i0 + u].columns;
                    const bool live = i0 + u < n && s_rec[warp][i0 + u].cell != 0u;
#pragma unroll
                    for (int k = 0; k < NV; ++k) {
                        g[u][k][0] = g[u][k][1] = 0ull;
                        if (live && ls.on[k])
                            load_quad<float>(p.columns + (static_cast<size_t>(from) + ls.column_at[k]) * 4, g[u][k]);
                    }
                }
                float t[U * 4];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int i = i0 + u;
                    if ((m_enter >> i) & 1u) {
                        const bool right = (m_right >> i) & 1u;
                        flush(0);
                        flush(2);
                        if (right) {
#pragma unroll
                            for (int c = 0; c < 4; c += 2)
#pragma unroll
                                for (int k = 0; k < NV; ++k)
#pragma unroll
                                    for (int e = 0; e < 2; ++e) {
                                        acc[c][k][e] = acc[c + 1][k][e];
                                        val[c][k][e] = val[c + 1][k][e];
                                        acc[c + 1][k][e] = 0ull;
                                    }
                        } else {
                            flush(1);
                            flush(3);
                        }
                        cur = s_rec[warp][i].row;
                        cell = s_rec[warp][i].cell;
                        if (!right) {
                            fetch(0);
                            fetch(2);
                        }
                        fetch(1);
                        fetch(3);
                    }
                    const Record& q = s_rec[warp][i];
                    const f32x2 w[4] = {q.w01.x, q.w01.y, q.w23.x, q.w23.y};
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        f32x2 dot = 0ull;
#pragma unroll
                        for (int k = 0; k < NV; ++k)
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                acc[c][k][e] = fma2(w[c], g[u][k][e], acc[c][k][e]);
                                dot = fma2(val[c][k][e], g[u][k][e], dot);
                            }
                        const float2 h = unpack2(dot);
                        t[u * 4 + c] = h.x + h.y;
                    }
                }
                // the sum of value v lands in the lanes of group v: gather a sample's four
                constexpr int N = U * 4, kShare = 32 / N;
                const float sum = reduce_values<N, 32>(t, lane);
                const int u = lane / (4 * kShare);
                float tc[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) tc[c] = __shfl_sync(0xffffffffu, sum, (u * 4 + c) * kShare);
                if (lane % (4 * kShare) < 3 && i0 + u < n) {
                    const Record& q = s_rec[warp][i0 + u];
                    const float hh = 1.f - q.lh, hw = 1.f - q.lw;
                    const int what = lane % (4 * kShare);   // mask, y, x
                    if (what == 0) {
                        if (p.grad_mask != nullptr) {
                            const float v = hh * (hw * tc[0] + q.lw * tc[1]) + q.lh * (hw * tc[2] + q.lw * tc[3]);
                            if (slices > 1) atomicAdd(p.grad_mask + q.id, v);
                            else p.grad_mask[q.id] = v;
                        }
                    } else {
                        const float v = q.mask * (what == 1 ? hw * (tc[2] - tc[0]) + q.lw * (tc[3] - tc[1])
                                                            : hh * (tc[1] - tc[0]) + q.lh * (tc[3] - tc[2]));
                        float* to = p.grad_offset + 2ull * q.id + (what - 1);
                        if (slices > 1) atomicAdd(to, v);
                        else *to = v;
                    }
                }
            }
            __syncwarp();
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) flush(c);
    }
}

size_t up(size_t v) { return (v + 255) / 256 * 256; }

}  // namespace

size_t sorted_bytes(const dcn_shape* s, const Derived& d) {
    const size_t items = static_cast<size_t>(d.M) * s->deform_groups * d.K;
    const size_t maps = static_cast<size_t>(s->N) * s->deform_groups;
    // 32-bit offsets, in quads; no more taps than the sort has threads (its Source::period)
    if (d.K > static_cast<int>(kSortThreads) || d.M * s->groups * d.Kd / 4 >= (1ll << 32) ||
        static_cast<long long>(s->N) * s->H * s->W * (s->C / 4) >= (1ll << 32) || items + maps >= (1ull << 28))
        return 0;
    return 256 + up(maps * sizeof(uint2)) + up(items * 4);
}

SortParams sorted_params(void* workspace, size_t items, uint32_t maps) {
    char* ws = static_cast<char*>(workspace);
    SortParams sp{};
    sp.ticket = reinterpret_cast<uint32_t*>(ws);
    sp.regions = reinterpret_cast<uint2*>(ws + 256);
    sp.sorted = reinterpret_cast<uint32_t*>(ws + 256 + up(maps * sizeof(uint2)));
    sp.nsamples = static_cast<uint32_t>(items);
    sp.nregions = maps;
    return sp;
}

// Tickets and grid of a main kernel whose samples are walked once per slice of the channels.
template <typename Kernel>
cudaError_t plan_slices(Kernel kern, int channels, const DcnParams& p, int sm_count, SortParams& sp,
                        uint32_t* slices, uint32_t* grid) {
    *slices = static_cast<uint32_t>((p.Cd + channels - 1) / channels);
    const LaunchShape shape{sm_count, 0};
    const void* k = reinterpret_cast<const void*>(kern);
    cudaError_t e = plan_tickets(k, 1, sp, static_cast<uint32_t>(p.HoWo) * p.K, shape, grid);
    int per_sm = 1;
    if (e == cudaSuccess) e = resident_ctas(k, kThreadsPerCta, 0, &per_sm);
    const unsigned long long want = static_cast<unsigned long long>(*grid) * *slices;
    const uint32_t cap = static_cast<uint32_t>(sm_count) * per_sm;
    *grid = want < cap ? static_cast<uint32_t>(want) : cap;
    return e;
}

int launch_gather_sorted(const DcnParams& p, void* workspace, long long M, int N, const ColumnsOut& to,
                         int sm_count, cudaStream_t stream) {
    const uint32_t maps = static_cast<uint32_t>(N) * p.DG;
    SortParams sp = sorted_params(workspace, static_cast<size_t>(M) * p.DG * p.K, maps);
    const uint32_t K = static_cast<uint32_t>(p.K);
    const uint32_t cells = static_cast<uint32_t>(p.H + 1) * static_cast<uint32_t>(p.W + 1) + 1u;
    const ConvSamples samples{p, static_cast<uint32_t>(p.HoWo) * K, K, static_cast<uint32_t>(p.DG) * K, cells, cells};
    cudaError_t e = launch_sort(samples, maps, sp, sm_count, stream);
    if (e != cudaSuccess) return note_cuda_error(e);
    auto launch = [&](auto kern, int channels) -> cudaError_t {
        uint32_t slices = 1, grid = 0;
        const cudaError_t err = plan_slices(kern, channels, p, sm_count, sp, &slices, &grid);
        if (err != cudaSuccess) return err;
        kern<<<grid, kThreadsPerCta, 0, stream>>>(p, sp, slices, to);
        return cudaGetLastError();
    };
    e = p.Cd > 128 ? launch(gather_sorted_kernel<2>, 256) : launch(gather_sorted_kernel<1>, 128);
    if (e != cudaSuccess) return note_cuda_error(e);
    count_launches(2);
    return MSDA_OK;
}

int launch_scatter_sorted(const DcnParams& p, const void* sorted, uint32_t* ticket, long long M, int N,
                          int sm_count, cudaStream_t stream) {
    const size_t items = static_cast<size_t>(M) * p.DG * p.K;
    SortParams sp = sorted_params(const_cast<void*>(sorted), items, static_cast<uint32_t>(N) * p.DG);
    sp.ticket = ticket;   // the regions and sample numbers are only read
    auto launch = [&](auto kern, int channels) -> cudaError_t {
        uint32_t slices = 1, grid = 0;
        cudaError_t err = plan_slices(kern, channels, p, sm_count, sp, &slices, &grid);
        if (err == cudaSuccess && slices > 1) {   // they add to these
            err = cudaMemsetAsync(p.grad_offset, 0, items * 8, stream);
            if (err == cudaSuccess && p.grad_mask != nullptr)
                err = cudaMemsetAsync(p.grad_mask, 0, items * 4, stream);
        }
        if (err != cudaSuccess) return err;
        kern<<<grid, kThreadsPerCta, 0, stream>>>(p, sp, slices);
        return cudaGetLastError();
    };
    const cudaError_t e =
        p.Cd > 128 ? launch(scatter_sorted_kernel<2>, 256) : launch(scatter_sorted_kernel<1>, 128);
    if (e != cudaSuccess) return note_cuda_error(e);
    count_launches(1);
    return MSDA_OK;
}

}  // namespace dcn
