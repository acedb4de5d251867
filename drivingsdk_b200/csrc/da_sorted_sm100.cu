// Deformable aggregation, backward over cell-sorted samples (cell_sort.cuh), for sm_100a.
//
// For a sample (anchor, point, camera, scale) with bilinear weights b_c on corner rows V_c and the
// group weights w of its channels:
//     grad_feat[V_c]  += b_c * (w * grad_out)          grad_w[group] = <sum_c b_c V_c, grad_out>_group
//     grad_loc        += size * <differences of the V_c, w * grad_out>
// A feature row is C channels (1 KB for 256), so per sample the task-ordered backward (da_sm100.cu)
// moves 4 KB each way between L2 and an SM. Sorted by cell, corner rows and their gradient sums
// stay in registers while the samples of a cell pass, and a sample costs its 1 KB of grad_out.
// One sample at a time per warp: lane = channel quads j and j + 32, all four corners.
#include "cell_sort.cuh"
#include "da_params.h"
#include "msda_tile.cuh"

namespace msda {

// Divisions that take a sample number apart.
struct DaDivs {
    FastDiv scales, cams, pts, anchors;
};

// What the sort needs to know: a map is one (batch, camera, scale), its samples are the (anchor,
// point) pairs.
template <typename T>
struct AggregationSamples {
    static constexpr uint32_t kInFlight = 4;   // samples in flight per thread of the sort
    static constexpr bool kMapsAlike = false;   // scales differ
    DaParams p;
    DaDivs fd;
    uint32_t samples;   // of one map: A * Pts
    uint32_t period, period_step;   // 1, cams * scales
    uint32_t most_cells, mean_cells;   // of a map

    struct Map {
        uint32_t cells, first;
        int W, H;
    };
    __device__ __forceinline__ bool ok() const { return true; }
    __device__ __forceinline__ Map map(uint32_t m) const {
        const uint32_t maps = static_cast<uint32_t>(p.cams) * p.scales;
        const uint32_t cs = m % maps, b = m / maps;
        Map r;
        r.H = p.use_table ? p.lv_h[cs] : p.shapes_dev[2 * cs];
        r.W = p.use_table ? p.lv_w[cs] : p.shapes_dev[2 * cs + 1];
        r.cells = static_cast<uint32_t>(r.H + 1) * static_cast<uint32_t>(r.W + 1);
        r.first = b * samples * maps + cs;
        return r;
    }
    __device__ __forceinline__ uint32_t id(const Map& m, uint32_t i) const {
        return m.first + i * (static_cast<uint32_t>(p.cams) * p.scales);
    }
    __device__ __forceinline__ float2 position(uint32_t id) const {
        return load_pair(reinterpret_cast<const T*>(p.loc) + 2ull * fd_div(id, fd.scales));
    }
    __device__ __forceinline__ uint32_t cell(const Map& m, float2 xy) const {
        const bool inside = xy.x > 0.f && xy.x < 1.f && xy.y > 0.f && xy.y < 1.f;
        return inside ? sample_cell<4>(xy, m.W, m.H) : kNoRow;
    }
    // all gradients start from zero
    __host__ __device__ void* sums() const { return p.grad_feat; }
    __host__ __device__ size_t sums_bytes() const { return static_cast<size_t>(p.B) * p.F * p.C * sizeof(float); }
    __host__ __device__ size_t points() const { return static_cast<size_t>(p.B) * p.A * p.Pts * p.cams; }
    __host__ __device__ size_t weight_bytes() const { return points() * p.scales * p.G * sizeof(float); }
    size_t clear_size() const { return points() * 8 + weight_bytes(); }
    __device__ __forceinline__ void clear(size_t first, size_t step) const {
        clear_bytes(p.grad_loc, points() * 8, first, step);
        clear_bytes(p.grad_wts, weight_bytes(), first, step);
    }
};

template <typename T, int NV>
__global__ void __launch_bounds__(kThreadsPerCta, 2)
da_bwd_sorted_kernel(const __grid_constant__ DaParams p, const __grid_constant__ DaDivs fd,
                     const __grid_constant__ SortParams sp) {
    constexpr int U = 2;   // samples in flight
    struct Record {
        ulonglong2 w01, w23;         // bilinear weights, each twice (packed multiply-add)
        float lw, lh, wf, hf;
        uint32_t go, row, cell, id;  // offsets of the grad_out and top-left rows; width << 4 | corners
    };
    __shared__ float4 s_map[kDaMaxMaps];   // width, height, width (bits), first row (bits)
    __shared__ __align__(16) Record s_rec[kWarpsPerCta][32];
    for (int i = threadIdx.x; i < p.cams * p.scales; i += blockDim.x) {
        const int h = p.use_table ? p.lv_h[i] : p.shapes_dev[2 * i];
        const int w = p.use_table ? p.lv_w[i] : p.shapes_dev[2 * i + 1];
        const int start = p.use_table ? p.lv_start[i] : p.starts_dev[i];
        s_map[i] = make_float4(static_cast<float>(w), static_cast<float>(h), __int_as_float(w),
                               __int_as_float(start));
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t units = p.row_units;      // quads per row
    const T* feat = reinterpret_cast<const T*>(p.feat) + lane * 4;
    const T* gout = reinterpret_cast<const T*>(p.grad_out) + lane * 4;
    const T* wts = reinterpret_cast<const T*>(p.wts);
    float* gfeat = p.grad_feat + lane * 4;
    const int qpg = p.cpg / 4;               // quads (lanes) per group: a power of two
    bool on[NV];
    int grp[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        on[k] = static_cast<uint32_t>(lane + 32 * k) < units;
        grp[k] = min((lane + 32 * k) / qpg, p.G - 1);
    }

    Ticket ticket;
    while (next_ticket(sp, sp.stream, lane, ticket)) {
        if (ticket.begin >= ticket.end) continue;
        f32x2 acc[4][NV][2], val[4][NV][2];
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int k = 0; k < NV; ++k) acc[c][k][0] = acc[c][k][1] = val[c][k][0] = val[c][k][1] = 0ull;
        uint32_t cur = 0u, cell = 0u;        // no corner: nothing to flush
        auto offset = [&](int c) {
            return static_cast<size_t>(cur + ((c & 1) ? units : 0u) + ((c & 2) ? (cell >> 4) * units : 0u)) * 4;
        };
        auto flush = [&](int c) {
            if ((cell >> c) & 1u) {
#pragma unroll
                for (int k = 0; k < NV; ++k)
                    if (on[k]) red_quad(gfeat + offset(c) + k * 128, acc[c][k]);
            }
#pragma unroll
            for (int k = 0; k < NV; ++k) acc[c][k][0] = acc[c][k][1] = 0ull;
        };
        auto fetch = [&](int c) {
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                val[c][k][0] = val[c][k][1] = 0ull;
                if (((cell >> c) & 1u) && on[k]) load_quad<T>(feat + offset(c) + k * 128, val[c][k]);
            }
        };
        for (uint32_t at = ticket.begin; at < ticket.end; at += 32) {
            // ---- lane = sample: cell, corner weights --------------------------------------
            const int n = min(32, static_cast<int>(ticket.end - at));
            Record r;
            r.go = r.row = r.cell = r.id = 0u;
            r.lw = r.lh = r.wf = r.hf = 0.f;
            r.w01 = r.w23 = make_ulonglong2(0ull, 0ull);
            if (lane < n) {
                r.id = __ldg(sp.sorted + at + lane);
                const uint32_t li = fd_div(r.id, fd.scales);
                const uint32_t pt = fd_div(li, fd.cams);
                const uint32_t row = fd_div(pt, fd.pts);          // b * A + anchor
                const uint32_t b = fd_div(row, fd.anchors);
                const float4 m = s_map[(li - pt * p.cams) * p.scales + (r.id - li * p.scales)];
                const int W = __float_as_int(m.z);
                const float2 xy = load_pair(reinterpret_cast<const T*>(p.loc) + 2ull * li);
                const float x0f = floorf(xy.x * m.x - 0.5f), y0f = floorf(xy.y * m.y - 0.5f);
                r.lw = fmaf(xy.x, m.x, -(x0f + 0.5f));
                r.lh = fmaf(xy.y, m.y, -(y0f + 0.5f));
                r.wf = m.x;
                r.hf = m.y;
                const float hw = 1.f - r.lw, hh = 1.f - r.lh;
                const uint32_t sides = (x0f >= 0.f ? 1u : 0u) | (x0f < m.x - 1.f ? 2u : 0u);
                r.cell = (static_cast<uint32_t>(W) << 4) | (y0f >= 0.f ? sides : 0u) |
                         (y0f < m.y - 1.f ? sides << 2 : 0u);
                r.row = (b * static_cast<uint32_t>(p.F) + __float_as_uint(m.w) +
                         static_cast<uint32_t>(__float2int_rz(y0f) * W + __float2int_rz(x0f))) * units;
                r.go = row * units;
                r.w01 = make_ulonglong2(pack2(hh * hw, hh * hw), pack2(hh * r.lw, hh * r.lw));
                r.w23 = make_ulonglong2(pack2(r.lh * hw, r.lh * hw), pack2(r.lh * r.lw, r.lh * r.lw));
            }
            uint32_t prow = __shfl_up_sync(0xffffffffu, r.row, 1);
            uint32_t pcell = __shfl_up_sync(0xffffffffu, r.cell, 1);
            if (lane == 0) {
                prow = cur;
                pcell = cell;
            }
            const uint32_t m_enter =
                __ballot_sync(0xffffffffu, lane < n && (r.row != prow || r.cell != pcell));
            const uint32_t m_right = __ballot_sync(
                0xffffffffu, r.row == prow + units && (r.cell >> 4) == (pcell >> 4) &&
                                 ((pcell >> 1) & 5u) == (r.cell & 5u));
            s_rec[warp][lane] = r;
            __syncwarp();

            // ---- warp = sample --------------------------------------------------------------
#pragma unroll 1
            for (int i0 = 0; i0 < n; i0 += U) {
                f32x2 go[U][NV][2];
                float w[U][NV];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    // past the last sample of an odd round: the record of nothing (zero weights)
                    const Record& q = s_rec[warp][i0 + u];
                    const bool live = i0 + u < n;
#pragma unroll
                    for (int k = 0; k < NV; ++k) {
                        go[u][k][0] = go[u][k][1] = 0ull;
                        w[u][k] = 0.f;
                        if (live && on[k]) {
                            load_quad<T>(gout + static_cast<size_t>(q.go) * 4 + k * 128, go[u][k]);
                            w[u][k] = Elem<T>::to_f(__ldg(wts + static_cast<size_t>(q.id) * p.G + grp[k]));
                        }
                    }
                }
                float d_loc[U][2], d_w[U][NV];
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
                    const f32x2 b[4] = {q.w01.x, q.w01.y, q.w23.x, q.w23.y};
                    f32x2 t[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll
                    for (int k = 0; k < NV; ++k) {
                        const f32x2 w2 = pack2(w[u][k], w[u][k]);
                        f32x2 dot = 0ull;
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const f32x2 wg = mul2(w2, go[u][k][e]);
                            f32x2 mean = 0ull;
#pragma unroll
                            for (int c = 0; c < 4; ++c) {
                                acc[c][k][e] = fma2(b[c], wg, acc[c][k][e]);
                                t[c] = fma2(val[c][k][e], wg, t[c]);
                                mean = fma2(b[c], val[c][k][e], mean);
                            }
                            dot = fma2(mean, go[u][k][e], dot);
                        }
                        const float2 h = unpack2(dot);
                        d_w[u][k] = h.x + h.y;
                    }
                    float tc[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        // (a corner outside the map: zeros, whose product with an infinite grad_out
                        // is not a number)
                        const float2 h = unpack2(t[c]);
                        tc[c] = ((cell >> c) & 1u) ? h.x + h.y : 0.f;
                    }
                    d_loc[u][0] = q.wf * ((1.f - q.lh) * (tc[1] - tc[0]) + q.lh * (tc[3] - tc[2]));
                    d_loc[u][1] = q.hf * ((1.f - q.lw) * (tc[2] - tc[0]) + q.lw * (tc[3] - tc[1]));
                }
                // location gradients over all lanes, weight gradients over a group's lanes
                float part[2 * U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    part[2 * u] = d_loc[u][0];
                    part[2 * u + 1] = d_loc[u][1];
                }
                const float loc_sum = reduce_values<2 * U, 32>(part, lane);
                for (int o = qpg >> 1; o >= 1; o >>= 1) {
#pragma unroll
                    for (int u = 0; u < U; ++u)
#pragma unroll
                        for (int k = 0; k < NV; ++k)
                            d_w[u][k] += __shfl_xor_sync(0xffffffffu, d_w[u][k], o);
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (i0 + u >= n) break;
                    const uint32_t id = s_rec[warp][i0 + u].id;
#pragma unroll
                    for (int k = 0; k < NV; ++k)
                        if (on[k] && (lane & (qpg - 1)) == 0)
                            p.grad_wts[static_cast<size_t>(id) * p.G + grp[k]] = d_w[u][k];
                }
                constexpr int kShare = 32 / (2 * U);
                const int v = lane / kShare;   // this lane's sum: sample v / 2, coordinate v % 2
                if (lane % kShare == 0 && i0 + v / 2 < n)
                    atomicAdd(p.grad_loc + 2ull * fd_div(s_rec[warp][i0 + v / 2].id, fd.scales) + v % 2,
                              loc_sum);
            }
            __syncwarp();
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) flush(c);
    }
}

template <typename T>
static cudaError_t launch_da_sorted(const DaParams& p, SortParams sp, int sm_count, cudaStream_t stream) {
    const uint32_t samples = static_cast<uint32_t>(p.A) * p.Pts;
    const DaDivs fd{make_fastdiv(p.scales), make_fastdiv(p.cams), make_fastdiv(p.Pts), make_fastdiv(p.A)};
    const uint32_t maps = static_cast<uint32_t>(p.cams) * p.scales, F = static_cast<uint32_t>(p.F);
    cudaError_t e = launch_sort(AggregationSamples<T>{p, fd, samples, 1u, maps, 2u * (F + 1u), F / maps},
                                static_cast<uint32_t>(p.B) * maps, sp, sm_count, stream);
    if (e != cudaSuccess) return e;
    const LaunchShape ls{sm_count, 0};
    auto launch = [&](auto kern) -> cudaError_t {
        uint32_t grid = 0;
        e = plan_tickets(reinterpret_cast<const void*>(kern), 1, sp, samples, ls, &grid);
        if (e != cudaSuccess) return e;
        kern<<<grid, kThreadsPerCta, 0, stream>>>(p, fd, sp);
        return cudaGetLastError();
    };
    return p.C > 128 ? launch(da_bwd_sorted_kernel<T, 2>) : launch(da_bwd_sorted_kernel<T, 1>);
}

cudaError_t launch_da_backward_sorted(const DaParams& p, SortParams sp, int dtype, int sm_count,
                                      cudaStream_t stream) {
    switch (dtype) {
        case 0: return launch_da_sorted<float>(p, sp, sm_count, stream);
        case 1: return launch_da_sorted<__half>(p, sp, sm_count, stream);
        case 2: return launch_da_sorted<__nv_bfloat16>(p, sp, sm_count, stream);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace msda
