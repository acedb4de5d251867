// Backward over samples sorted by the pixel cell they fall into, shared by the bilinear operator
// (MSDA, CPS = 4 corners per sample) and the nearest-pixel operator (CPS = 1).
//
// The task-ordered backward (msda_bwd_kernel.cuh) gathers and reduces every corner row of every
// sample: 8 row transfers between L2 and an SM per sample, of which the reductions retire at
// the sector rate of L2. Samples of one cell share their four corner rows. Walking the samples
// cell by cell keeps the corner rows and their gradient sums in registers, and what is left per
// sample is one row of grad_out; corner rows are loaded and their sums reduced once per run of
// samples in a cell (and only the new two when the walk moves one cell to the right).
//
//   1 sort     cluster of CTAs = (batch, head, level): counting sort by cell in shared memory;
//              zeros for all that the main kernel adds to or may leave out.
//   2 main     warp = a ticket of consecutive sorted samples, in 32 / LPR streams: a stream is
//              LPR lanes, each lane four channels of all corners.
// The main kernel compares the cells themselves, so the order is only a matter of speed.
// Work is cut by samples, not by cells: a map whose samples all fall into one cell is as
// balanced as any other.
#pragma once

#include <type_traits>

#include "cell_sort.cuh"
#include "msda_tile.cuh"

namespace msda {

// Level table of one CTA.
struct SortLevels {
    float4 geo[kMaxLevels];   // width, height, width (bits), first key (bits)
};

// All threads of the CTA must call it. False: a level table in device memory is inconsistent
// (status bit set); nothing may be touched then.
__device__ __forceinline__ bool load_sort_levels(const Params& p, SortLevels& lv) {
    if (!device_level_table_ok(p)) return false;
    for (int l = threadIdx.x; l < p.L; l += blockDim.x) {
        const int h = p.use_table ? p.lv.h[l] : p.shapes_dev[2 * l * p.table_step];
        const int w = p.use_table ? p.lv.w[l] : p.shapes_dev[(2 * l + 1) * p.table_step];
        const int start = p.use_table ? p.lv.start[l] : p.start_dev[l * p.table_step];
        lv.geo[l] = make_float4(static_cast<float>(w), static_cast<float>(h), __int_as_float(w),
                                __int_as_float(start));
    }
    __syncthreads();
    return true;
}

// Task, level and sample-in-task of sample number `id`.
struct SampleId {
    uint32_t task, b, h;
    int level;
};
__device__ __forceinline__ SampleId sample_id(const Params& p, const SortParams& sp, uint32_t id) {
    SampleId r;
    r.task = fd_div(id, p.fd_lp);
    r.level = static_cast<int>(fd_div(id - r.task * p.LP, sp.fd_p));
    r.b = fd_div(r.task, p.fd_qh);
    r.h = r.task - fd_div(r.task, p.fd_h) * p.H;
    return r;
}

// What the sort needs to know (cell_sort.cuh): a map is one (batch, head, level).
template <typename TL, int CPS>
struct AttentionSamples {
    static constexpr uint32_t kInFlight = 4;   // samples in flight per thread of the sort
    static constexpr bool kMapsAlike = false;   // levels differ
    Params p;
    FastDiv fd_p;       // division by the points per level
    uint32_t samples;   // of one map: Q * P
    uint32_t period, period_step;   // the numbers of samples that many apart differ by period_step
    uint32_t most_cells, mean_cells;   // of a map

    struct Map {
        uint32_t cells, first;   // first: number of the map's first sample
        int W, H;
    };
    __device__ __forceinline__ bool ok() const { return device_level_table_ok(p); }
    __device__ __forceinline__ Map map(uint32_t m) const {
        const uint32_t l = m % p.L, bh = m / p.L;
        const uint32_t h = bh % p.H, b = bh / p.H;
        Map r;
        r.H = p.use_table ? p.lv.h[l] : p.shapes_dev[2 * l * p.table_step];
        r.W = p.use_table ? p.lv.w[l] : p.shapes_dev[(2 * l + 1) * p.table_step];
        r.cells = (CPS == 4) ? static_cast<uint32_t>(r.H + 1) * static_cast<uint32_t>(r.W + 1)
                             : static_cast<uint32_t>(r.H) * static_cast<uint32_t>(r.W);
        r.first = (b * p.Q * p.H + h) * p.LP + l * p.P;
        return r;
    }
    // sample i of the map: point i % P of query i / P
    __device__ __forceinline__ uint32_t id(const Map& m, uint32_t i) const {
        const uint32_t q = fd_div(i, fd_p);
        return m.first + q * (static_cast<uint32_t>(p.H) * p.LP) + (i - q * p.P);
    }
    __device__ __forceinline__ float2 position(uint32_t id) const {
        return load_pair(static_cast<const TL*>(p.loc) + 2ull * id);
    }
    __device__ __forceinline__ uint32_t cell(const Map& m, float2 xy) const {
        return sample_cell<CPS>(xy, m.W, m.H);
    }
    // What starts from zero: the sums of value's gradient ...
    __host__ __device__ void* sums() const { return p.grad_value; }
    __host__ __device__ size_t sums_bytes() const {
        return static_cast<size_t>(p.B) * p.K * p.H * p.D * sizeof(float);
    }
    // ... and the gradients of locations and weights, since a sample that takes no part has none (zeros
    // for the dropped samples alone, a few bytes each, cost 55 us where 28 % of 20 M are dropped).
    __host__ __device__ size_t samples_bytes() const {   // of one number per sample
        return CPS == 4 ? static_cast<size_t>(p.ntasks) * p.LP * sizeof(TL) : 0;
    }
    size_t clear_size() const { return 3 * samples_bytes(); }
    __device__ __forceinline__ void clear(size_t first, size_t step) const {
        if constexpr (CPS == 4) {
            clear_bytes(p.grad_loc, 2 * samples_bytes(), first, step);
            clear_bytes(p.grad_attn, samples_bytes(), first, step);
        }
    }
};

// ---------------------------------------------------------------------------
// main kernels
// ---------------------------------------------------------------------------
// One sorted sample, on its lane.
struct SortedSample {
    uint32_t row;    // row offset of the cell's top-left corner (wraps where that does not exist)
    uint32_t cell;   // level width << 4 | existing corners
    uint32_t task, id;
    float lw, lh, a, wf, hf;
    float w[4];
    bool amplified;
};
// MSDA_DEBUG_BOUNDS build: the rows of the cell's existing corners against the extent of value and
// grad_value (see debug_check_rows); an offending sample loses all its corners.
__device__ __forceinline__ void debug_check_cell(const Params& p, SortedSample& s) {
#ifdef MSDA_DEBUG_BOUNDS
    const uint32_t step_x = static_cast<uint32_t>(p.H) * p.row_units;
    bool bad = false;
    for (int c = 0; c < 4; ++c) {
        const uint32_t off = s.row + ((c & 1) ? step_x : 0u) + ((c & 2) ? (s.cell >> 4) * step_x : 0u);
        bad |= ((s.cell >> c) & 1u) && (off >= p.limit_units || p.limit_units - off < p.row_units);
    }
    if (bad) {
        atomicOr(p.status, kStatusOutOfBounds);
        s.cell &= ~15u;
    }
#else
    (void)p;
    (void)s;
#endif
}

// What a lane loads for a sample; fetched a round ahead of its use.
struct RawSample {
    uint32_t id;
    float2 xy;
    float a;
};
template <typename TL>
__device__ __forceinline__ void load_raw(const Params& p, RawSample& r, bool live) {
    r.xy = make_float2(0.f, 0.f);
    r.a = 0.f;
    if (live) {
        r.xy = load_pair(static_cast<const TL*>(p.loc) + 2ull * r.id);
        r.a = Elem<TL>::to_f(__ldg(static_cast<const TL*>(p.attn) + r.id));
    }
}
template <int CPS>
__device__ __forceinline__ SortedSample set_up_sample(const Params& p, const SortParams& sp,
                                                      const SortLevels& lv, const RawSample& raw,
                                                      bool live) {
    SortedSample r;
    r.row = r.cell = r.task = r.id = 0u;   // no corner, task 0: adds nothing
    r.lw = r.lh = r.a = r.wf = r.hf = 0.f;
    r.w[0] = r.w[1] = r.w[2] = r.w[3] = 0.f;
    r.amplified = false;
    if (!live) return r;
    r.id = raw.id;
    const SampleId s = sample_id(p, sp, r.id);
    const float4 geo = lv.geo[s.level];
    const int W = __float_as_int(geo.z);
    const uint32_t row_base =
        (s.b * static_cast<uint32_t>(p.K) + __float_as_uint(geo.w)) * p.H + s.h;
    r.task = s.task;
    r.a = raw.a;
    r.wf = geo.x;
    r.hf = geo.y;
    if constexpr (CPS == 4) {
        // sample_setup (msda_common.cuh) for a sample known to take part
        const float x0f = floorf(raw.xy.x * geo.x - 0.5f);
        const float y0f = floorf(raw.xy.y * geo.y - 0.5f);
        r.lw = fmaf(raw.xy.x, geo.x, -(x0f + 0.5f));
        r.lh = fmaf(raw.xy.y, geo.y, -(y0f + 0.5f));
        const float hw = 1.f - r.lw, hh = 1.f - r.lh;
        const uint32_t sides = (x0f >= 0.f ? 1u : 0u) | (x0f < geo.x - 1.f ? 2u : 0u);
        r.cell = (static_cast<uint32_t>(W) << 4) | (y0f >= 0.f ? sides : 0u) |
                 (y0f < geo.y - 1.f ? sides << 2 : 0u);
        r.row = (row_base + static_cast<uint32_t>(__float2int_rz(y0f) * W + __float2int_rz(x0f)) * p.H) *
                p.row_units;
        const float top = hh * r.a, bottom = r.lh * r.a;
        r.w[0] = top * hw;
        r.w[1] = top * r.lw;
        r.w[2] = bottom * hw;
        r.w[3] = bottom * r.lw;
        r.amplified = fmaxf(geo.x, geo.y) * fabsf(r.a) >= p.precise_amp;
    } else {
        const int x = min(max(__float2int_rz(raw.xy.x), 0), W - 1);
        const int y = min(max(__float2int_rz(raw.xy.y), 0), __float2int_rz(geo.y) - 1);
        r.row = (row_base + static_cast<uint32_t>(y * W + x) * p.H) * p.row_units;
        r.cell = 1u;
    }
    debug_check_cell(p, r);
    return r;
}
// Flags of a sorted sample in its stream (low bits; level width << 8 and existing corners << 4
// above them).
constexpr uint32_t kEnters = 1;      // its cell is not the previous sample's
constexpr uint32_t kJumps = 2;       // ... and not the next one to the right either
constexpr uint32_t kAmplified = 4;   // its dot products are formed in double

// Rows of grad_out in flight per lane and CTAs per SM. The kernel waits for the latency of its own
// instructions more than for memory (with grad_out from L1 it is no faster): at 80 registers and three CTAs
// two rows, more where two CTAs are as fast. Measured (us, main kernel):
//   128 channels, 16 bit, 20.5 M samples   2 rows x 3 CTAs 1820   4 x 2 1772   8 x 2 1622
//   128 channels, fp32, 4.6 M               630   617   1009 (spills)
//    64 channels, fp32, 5.1 M               378   394    673
//    32 channels, fp32, 4.6 M               265   267    358
//    16 channels, fp32, 5.1 M               196   173      -
// SPARSE: 16-bit rows that leave some of 32 lanes idle enter cells more slowly with eight rows than with two
// (whole backward, 96 channels, bf16: 1.65 M samples, 4 per cell 450 / 376; 1.39 M, 13 per cell 238 / 222;
// 5.1 M, 21 per cell 656 / 644; 2.56 M, 143 per cell 288 / 312; where most samples fall outside their
// map fewer share a cell than the number says: 80 channels, 4.9 M, 23 per cell 507 / 433).
template <typename T, int NV, int LPR, bool SPARSE>
struct SortedTile {
    static constexpr bool kMore = NV == 1 && (LPR == 32 || LPR == 4) && !SPARSE;
    static constexpr int kRows = !kMore ? 2 : (LPR == 32 && sizeof(T) == 2) ? 8 : 4;
    static constexpr int kCtas = (kMore || NV > 1) ? 2 : 3;
};

// Bilinear main kernel. T: type of value / grad_out; TL: type of locations, weights and their
// gradients. LPR lanes cover a row (4 channels each, NV times; lanes past D are idle, D need not
// be a power of two) and hold all four corners of a cell: value rows and gradient sums. A warp
// walks 32 / LPR streams of sp.stream consecutive sorted samples side by side, in rounds of 32
// samples whose set-up and final gradients are done lane = sample. The accumulation rows are
// fp32. RAGGED: some of those lanes are past D; without their checks the rest is 1 to 4 % faster
// (encoder shape, fp32, 32 channels: 284 -> 274 us; 128 channels, bf16: 1894 -> 1867 us).
template <typename T, typename TL, int NV, int LPR, bool RAGGED, bool SPARSE>
__global__ void __launch_bounds__(kThreadsPerCta, SortedTile<T, NV, LPR, SPARSE>::kCtas)
msda_bwd_sorted_kernel(const __grid_constant__ Params p, const __grid_constant__ SortParams sp) {
    constexpr int S = 32 / LPR;       // streams
    constexpr int U = SortedTile<T, NV, LPR, SPARSE>::kRows;   // rows of grad_out in flight per lane
    // fp32 bilinear operator: some dot products need double precision (see sample_grad)
    constexpr bool WIDE = sizeof(TL) == 4 && sizeof(T) == 4;
    static_assert(LPR % U == 0, "a round is LPR steps");

    __shared__ SortLevels lv;
    // records of one round, stream index fastest (streams then read different banks):
    // weights, each twice (operands of the packed multiply-add), later the dot products; those
    // formed in double; offset of the grad_out row and flags; row offset of the top-left corner
    __shared__ ulonglong2 s_w[kWarpsPerCta][32][2];
    __shared__ double s_wide[WIDE ? kWarpsPerCta : 1][WIDE ? 32 : 1][4];
    __shared__ uint2 s_rec[kWarpsPerCta][32];
    __shared__ uint32_t s_row[kWarpsPerCta][32];
    // what a lane needs of its sample after the products, out of the way of their registers
    struct Parked {
        uint32_t id, cell;
        float lw, lh, a, wf, hf;
        uint32_t amplified;
    };
    __shared__ __align__(16) Parked s_park[kWarpsPerCta][32];
    if (!load_sort_levels(p, lv)) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane / LPR, j = lane % LPR;
    const int my_stream = lane % S, my_step = lane / S;   // of this lane's sample in a round

    const uint32_t step_x = static_cast<uint32_t>(p.H) * p.row_units;
    bool on[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) on[k] = !RAGGED || (j + k * LPR) * 4 < p.D;
    const T* vlane = static_cast<const T*>(p.value) + j * 4;
    const T* glane = static_cast<const T*>(p.grad_out) + j * 4;
    float* alane = static_cast<float*>(p.grad_value) + j * 4;
    const uint32_t ticket_len = sp.stream * S;

    Ticket ticket;
    while (next_ticket(sp, ticket_len, lane, ticket)) {
        if (ticket.begin >= ticket.end) continue;
        f32x2 acc[4][NV][2], val[4][NV][2];
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int k = 0; k < NV; ++k) acc[c][k][0] = acc[c][k][1] = val[c][k][0] = val[c][k][1] = 0ull;
        // cell of this lane's stream and the offset of the pixel row below it; no corner: nothing
        // to flush
        uint32_t cur = 0u, cell = 0u, below = 0u;

        auto flush = [&](int c, bool yes) {
            if (yes && ((cell >> c) & 1u)) {
                float* at = alane + static_cast<size_t>(cur + ((c & 1) ? step_x : 0u) +
                                                        ((c & 2) ? below : 0u)) * 4;
#pragma unroll
                for (int k = 0; k < NV; ++k)
                    if (on[k]) red_quad(at + k * (LPR * 4), acc[c][k]);
            }
        };
        auto fetch = [&](int c, bool yes) {
            if (yes) {
                const T* at = vlane + static_cast<size_t>(cur + ((c & 1) ? step_x : 0u) +
                                                          ((c & 2) ? below : 0u)) * 4;
#pragma unroll
                for (int k = 0; k < NV; ++k) {
                    val[c][k][0] = val[c][k][1] = 0ull;
                    if (((cell >> c) & 1u) && on[k]) load_quad<T>(at + k * (LPR * 4), val[c][k]);
                }
            }
        };
        auto clear = [&](int c, bool yes) {
            if (yes) {
#pragma unroll
                for (int k = 0; k < NV; ++k) acc[c][k][0] = acc[c][k][1] = 0ull;
            }
        };
        // right corners become left ones
        auto shift = [&](int c, bool yes) {
            if (yes) {
#pragma unroll
                for (int k = 0; k < NV; ++k)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        acc[c][k][e] = acc[c + 1][k][e];
                        val[c][k][e] = val[c + 1][k][e];
                    }
            }
        };

        // this lane's samples: at, at + LPR, ... below `end`
        uint32_t at = ticket.begin + my_stream * sp.stream + my_step;
        const uint32_t end = min(ticket.end, ticket.begin + (my_stream + 1) * sp.stream);
        RawSample raw;
        raw.id = at < end ? __ldg(sp.sorted + at) : 0u;
        uint32_t next_id = at + LPR < end ? __ldg(sp.sorted + at + LPR) : 0u;
        load_raw<TL>(p, raw, at < end);
        for (; __any_sync(0xffffffffu, at < end); at += LPR) {
            // ---- lane = sample: cell, corner weights --------------------------------------
            RawSample next;
            next.id = next_id;
            load_raw<TL>(p, next, at + LPR < end);
            next_id = at + 2 * LPR < end ? __ldg(sp.sorted + at + 2 * LPR) : 0u;
            // Bit = lane = (step, stream) of the round. Not with two quads per lane: there a warp is one stream,
            // whose flags all lanes hold, and the masks cost spills (256 channels, fp32, 4.7 M samples:
            // 1328 us with them, 1119 without).
            uint32_t m_enter = 0u, m_jump = 0u, m_wide = 0u;
            {
                const SortedSample s = set_up_sample<4>(p, sp, lv, raw, at < end);
                raw = next;
                s_park[warp][lane] = Parked{s.id, s.cell, s.lw, s.lh, s.a, s.wf, s.hf, s.amplified ? 1u : 0u};
                uint32_t prow = __shfl_up_sync(0xffffffffu, s.row, S);
                uint32_t pcell = __shfl_up_sync(0xffffffffu, s.cell, S);
                const uint32_t srow = __shfl_sync(0xffffffffu, cur, my_stream * LPR);
                const uint32_t scell = __shfl_sync(0xffffffffu, cell, my_stream * LPR);
                if (my_step == 0) {
                    prow = srow;
                    pcell = scell;
                }
                uint32_t flags = s.cell << 4;
                if (WIDE && s.amplified) flags |= kAmplified;
                if (s.row != prow || s.cell != pcell) {
                    const bool right = s.row == prow + step_x && (s.cell >> 4) == (pcell >> 4) &&
                                       ((pcell >> 1) & 5u) == (s.cell & 5u);
                    flags |= right ? kEnters : (kEnters | kJumps);
                }
                if constexpr (NV == 1) {
                    m_enter = __ballot_sync(0xffffffffu, flags & kEnters);
                    m_jump = __ballot_sync(0xffffffffu, flags & kJumps);
                    m_wide = WIDE ? __ballot_sync(0xffffffffu, s.amplified) : 0u;
                }
                s_w[warp][lane][0] = make_ulonglong2(pack2(s.w[0], s.w[0]), pack2(s.w[1], s.w[1]));
                s_w[warp][lane][1] = make_ulonglong2(pack2(s.w[2], s.w[2]), pack2(s.w[3], s.w[3]));
                s_rec[warp][lane] = make_uint2(s.task * p.row_units, flags);
                s_row[warp][lane] = s.row;
            }
            __syncwarp();

            // ---- lanes = (stream, four channels) ------------------------------------------
#pragma unroll 1
            for (int t0 = 0; t0 < LPR; t0 += U) {
                uint32_t flags[U];
                f32x2 go[U][NV][2];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint2 rec = s_rec[warp][(t0 + u) * S + g];
                    flags[u] = rec.y;
                    const T* row = glane + static_cast<size_t>(rec.x) * 4;
#pragma unroll
                    for (int k = 0; k < NV; ++k) {
                        go[u][k][0] = go[u][k][1] = 0ull;
                        if (on[k]) load_quad<T>(row + k * (LPR * 4), go[u][k]);
                    }
                }
                float d[U * 4];
                constexpr uint32_t kStep = (S == 32) ? 0xffffffffu : (1u << S) - 1u;   // bits of a step
                auto products = [&](int u) {
                    const int slot = (t0 + u) * S + g;
                    f32x2 w[4];
                    {
                        const ulonglong2 w01 = s_w[warp][slot][0], w23 = s_w[warp][slot][1];
                        w[0] = w01.x;
                        w[1] = w01.y;
                        w[2] = w23.x;
                        w[3] = w23.y;
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        f32x2 a2 = 0ull;
#pragma unroll
                        for (int k = 0; k < NV; ++k)
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                acc[c][k][e] = fma2(w[c], go[u][k][e], acc[c][k][e]);
                                a2 = (k + e == 0) ? mul2(val[c][k][e], go[u][k][e])
                                                  : fma2(val[c][k][e], go[u][k][e], a2);
                            }
                        const float2 h = unpack2(a2);
                        d[u * 4 + c] = h.x + h.y;
                    }
                };
                // Most often nothing but products: without a branch between them the steps overlap.
                const uint32_t here = (m_enter | m_wide) >> (t0 * S);
                if (NV == 1 && (here & ((1u << (U * S - 1) << 1) - 1u)) == 0u) {
#pragma unroll
                    for (int u = 0; u < U; ++u) products(u);
                } else {
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int slot = (t0 + u) * S + g;
                        static_assert(NV == 1 || S == 1, "flags speak for the whole step");
                        auto any = [&](uint32_t mask, uint32_t flag) {   // of the streams in this step
                            return (NV == 1 ? (mask >> ((t0 + u) * S)) & kStep : flags[u] & flag) != 0u;
                        };
                        if (any(m_enter, kEnters)) {
                            const bool enters = flags[u] & kEnters, jumps = flags[u] & kJumps;
                            const bool any_jumps = any(m_jump, kJumps);
                            flush(0, enters);
                            flush(2, enters);
                            if (any_jumps) {
                                flush(1, jumps);
                                flush(3, jumps);
                                clear(0, jumps);
                                clear(2, jumps);
                            }
                            shift(0, enters && !jumps);
                            shift(2, enters && !jumps);
                            clear(1, enters);
                            clear(3, enters);
                            cur = s_row[warp][slot];      // the same for a stream that stays
                            cell = flags[u] >> 4;
                            below = (cell >> 4) * step_x;
                            if (any_jumps) {
                                fetch(0, jumps);
                                fetch(2, jumps);
                            }
                            fetch(1, enters);
                            fetch(3, enters);
                        }
                        products(u);
                        if constexpr (WIDE) {
                            // A step with an amplified sample forms its dot products in double as
                            // well; each sample takes the kind it asked for, so its gradients do
                            // not depend on which samples share the step.
                            if (any(m_wide, kAmplified)) {
                                double dd[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
                                for (int k = 0; k < NV; ++k)
#pragma unroll
                                    for (int e = 0; e < 2; ++e) {
                                        const float2 gf = unpack2(go[u][k][e]);
                                        const double gx = gf.x, gy = gf.y;
#pragma unroll
                                        for (int c = 0; c < 4; ++c) {
                                            const float2 vf = unpack2(val[c][k][e]);
                                            dd[c] = fma(static_cast<double>(vf.x), gx, dd[c]);
                                            dd[c] = fma(static_cast<double>(vf.y), gy, dd[c]);
                                        }
                                    }
                                const double r = reduce_values<4, LPR>(dd, j);
                                if (j % (LPR / 4) == 0) s_wide[warp][slot][j / (LPR / 4)] = r;
                            }
                        }
                    }
                }
                __syncwarp();   // every lane has read the weights of these steps
                constexpr int N = (U * 4 < LPR) ? U * 4 : LPR;   // dot products per reduction
#pragma unroll
                for (int q = 0; q < U * 4 / N; ++q) {
                    float part[N];
#pragma unroll
                    for (int i = 0; i < N; ++i) part[i] = d[q * N + i];
                    const float r = reduce_values<N, LPR>(part, j);
                    if (j % (LPR / N) == 0) {
                        const int v = q * N + j / (LPR / N);
                        reinterpret_cast<float*>(s_w[warp][(t0 + v / 4) * S + g])[v % 4] = r;
                    }
                }
            }
            __syncwarp();

            // ---- lane = sample: gradients of location and weight ---------------------------
            if (at < end) {
                using Acc = typename std::conditional<WIDE, double, float>::type;
                const Parked s = s_park[warp][lane];
                const float4 h4 = *reinterpret_cast<const float4*>(s_w[warp][lane]);
                Acc S4[4] = {h4.x, h4.y, h4.z, h4.w};
                if constexpr (WIDE) {
                    if (s.amplified) {
#pragma unroll
                        for (int c = 0; c < 4; ++c) S4[c] = s_wide[warp][lane][c];
                    }
                }
                // a corner outside the map counts as zero whatever grad_out holds: its product of zeros
                // with an infinity is not a number
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (((s.cell >> c) & 1u) == 0u) S4[c] = Acc(0);
                const Acc lw = s.lw, lh = s.lh, wf = s.wf, hf = s.hf, a = s.a;
                const Acc hw = Acc(1) - lw, hh = Acc(1) - lh;
                const float ga = static_cast<float>(hh * hw * S4[0] + hh * lw * S4[1] +
                                                    lh * hw * S4[2] + lh * lw * S4[3]);
                const float gx = static_cast<float>(wf * a * (hh * (S4[1] - S4[0]) + lh * (S4[3] - S4[2])));
                const float gy = static_cast<float>(hf * a * (hw * (S4[2] - S4[0]) + lw * (S4[3] - S4[1])));
                store_pair(static_cast<TL*>(p.grad_loc) + 2ull * s.id, gx, gy);
                static_cast<TL*>(p.grad_attn)[s.id] = Elem<TL>::from_f(ga);
            }
            __syncwarp();
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) flush(c, true);
    }
}

// Nearest-pixel main kernel: one row per sample. LPR lanes cover a row (four channels each, NV
// times), 32 / LPR samples of one pixel are worked on at a time and share its row. Bound by shared memory
// and L1 and by its own chains together (64 % of the load/store wavefronts, 55 % of the issue slots; with
// grad_out rows from L1 7 % faster): records
// in shared memory instead of two shuffles per row, and no guards for groups within their pixel,
// took 10.3 M samples on 375 pixels, 64 channels, from 317 to 287 us (bf16 327 to 260).
template <typename T, typename TL, int NV, int LPR, bool RAGGED>
__global__ void __launch_bounds__(kThreadsPerCta, NV > 1 ? 2 : 4)
gka_bwd_sorted_kernel(const __grid_constant__ Params p, const __grid_constant__ SortParams sp) {
    constexpr int U = 4;            // rows of grad_out in flight per lane
    constexpr int SL = 32 / LPR;    // samples per step
    __shared__ SortLevels lv;
    __shared__ float s_dot[kWarpsPerCta][32];
    __shared__ uint2 s_rec[kWarpsPerCta][32];   // offset of the sample's grad_out row, weight
    if (!load_sort_levels(p, lv)) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int j = lane % LPR, g = lane / LPR;
    float* dot = s_dot[warp];
    bool on[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) on[k] = !RAGGED || (j + k * LPR) * 4 < p.D;
    const T* vlane = static_cast<const T*>(p.value) + j * 4;
    const T* glane = static_cast<const T*>(p.grad_out) + j * 4;
    float* alane = static_cast<float*>(p.grad_value) + j * 4;

    Ticket ticket;
    while (next_ticket(sp, sp.stream, lane, ticket)) {
        const uint32_t base = ticket.begin, end = ticket.end;
        if (base >= end) continue;
        f32x2 acc[NV][2], val[NV][2];
#pragma unroll
        for (int k = 0; k < NV; ++k) acc[k][0] = acc[k][1] = val[k][0] = val[k][1] = 0ull;
        uint32_t cur = 0u, cell = 0u;
        auto flush = [&]() {
            if (cell & 1u) {
#pragma unroll
                for (int k = 0; k < NV; ++k) {
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        float2 a = unpack2(acc[k][e]);
#pragma unroll
                        for (int o = LPR; o < 32; o <<= 1) {
                            a.x += __shfl_xor_sync(0xffffffffu, a.x, o);
                            a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
                        }
                        acc[k][e] = pack2(a.x, a.y);
                    }
                    if (g == 0 && on[k])
                        red_quad(alane + (static_cast<size_t>(cur) + k * LPR) * 4, acc[k]);
                }
            }
        };
        RawSample raw;
        raw.id = base + lane < end ? __ldg(sp.sorted + base + lane) : 0u;
        uint32_t next_id = base + 32 + lane < end ? __ldg(sp.sorted + base + 32 + lane) : 0u;
        load_raw<TL>(p, raw, base + lane < end);
        for (uint32_t at = base; at < end; at += 32) {
            const int n = min(32, static_cast<int>(end - at));
            RawSample next;
            next.id = next_id;
            load_raw<TL>(p, next, at + 32 + lane < end);
            next_id = at + 64 + lane < end ? __ldg(sp.sorted + at + 64 + lane) : 0u;
            const SortedSample s = set_up_sample<1>(p, sp, lv, raw, lane < n);
            raw = next;
            uint32_t prow = __shfl_up_sync(0xffffffffu, s.row, 1);
            uint32_t pcell = __shfl_up_sync(0xffffffffu, s.cell, 1);
            if (lane == 0) {
                prow = cur;
                pcell = cell;
            }
            const uint32_t m_other =
                __ballot_sync(0xffffffffu, lane < n && (s.row != prow || s.cell != pcell));
            s_rec[warp][lane] = make_uint2(s.task * p.row_units, __float_as_uint(s.a));
            __syncwarp();
            // U * SL samples of the pixel from i0 on; WHOLE: none of them lies past `last`
            auto products = [&](int i0, int last, auto whole_tag) {
                constexpr bool WHOLE = decltype(whole_tag)::value;
                f32x2 go[U][NV][2];
                float w[U], d[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int i = i0 + u * SL + g;
                    const bool live = WHOLE || i < last;
                    const uint2 rec = s_rec[warp][WHOLE ? i : min(i, 31)];
                    w[u] = live ? __uint_as_float(rec.y) : 0.f;
                    const T* row = glane + static_cast<size_t>(rec.x) * 4;
#pragma unroll
                    for (int k = 0; k < NV; ++k) {
                        if (!WHOLE || RAGGED) go[u][k][0] = go[u][k][1] = 0ull;
                        if (live && on[k]) load_quad<T>(row + k * (LPR * 4), go[u][k]);
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const f32x2 w2 = pack2(w[u], w[u]);
                    f32x2 a2 = 0ull;
#pragma unroll
                    for (int k = 0; k < NV; ++k)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            acc[k][e] = fma2(w2, go[u][k][e], acc[k][e]);
                            a2 = (k + e == 0) ? mul2(val[k][e], go[u][k][e])
                                              : fma2(val[k][e], go[u][k][e], a2);
                        }
                    const float2 h = unpack2(a2);
                    d[u] = h.x + h.y;
                }
                const float r = reduce_values<U, LPR>(d, j);
                const int i = i0 + (j / (LPR / U)) * SL + g;
                if (j % (LPR / U) == 0 && (WHOLE || i < last)) dot[i] = r;
            };
#pragma unroll 1
            for (int first = 0; first < n;) {
                // samples [first, last) share a pixel
                const uint32_t later = m_other & ~((2u << first) - 1u);
                const int last = later != 0u ? __ffs(later) - 1 : n;
                if ((m_other >> first) & 1u) {
                    flush();
                    cur = __shfl_sync(0xffffffffu, s.row, first);
                    cell = __shfl_sync(0xffffffffu, s.cell, first);
#pragma unroll
                    for (int k = 0; k < NV; ++k) {
                        acc[k][0] = acc[k][1] = val[k][0] = val[k][1] = 0ull;
                        if (on[k] && (cell & 1u))
                            load_quad<T>(vlane + (static_cast<size_t>(cur) + k * LPR) * 4, val[k]);
                    }
                }
                int i0 = first;
#pragma unroll 1
                for (; i0 + U * SL <= last; i0 += U * SL) products(i0, last, std::true_type{});
                if (i0 < last) products(i0, last, std::false_type{});
                first = last;
            }
            __syncwarp();
            if (lane < n) static_cast<TL*>(p.grad_attn)[s.id] = Elem<TL>::from_f(dot[lane]);
            __syncwarp();
        }
        flush();
    }
}

// ---------------------------------------------------------------------------
// launch
// ---------------------------------------------------------------------------
template <typename Kernel>
static cudaError_t launch_sorted_main(Kernel kern, int streams, const Params& p, SortParams sp,
                                      uint32_t samples_per_map, const LaunchShape& ls,
                                      cudaStream_t stream) {
    uint32_t grid = 0;
    const cudaError_t e = plan_tickets(reinterpret_cast<const void*>(kern), streams, sp,
                                       samples_per_map, ls, &grid);
    if (e != cudaSuccess) return e;
    kern<<<grid, kThreadsPerCta, 0, stream>>>(p, sp);
    return cudaGetLastError();
}

// The lanes of a row of D channels: launch(pieces per lane, lanes).
template <typename Launch>
static cudaError_t for_row_width(int D, const Launch& launch) {
    const std::integral_constant<int, 1> one;
    if (D <= 16) return launch(one, std::integral_constant<int, 4>());
    if (D <= 32) return launch(one, std::integral_constant<int, 8>());
    if (D <= 64) return launch(one, std::integral_constant<int, 16>());
    if (D <= 128) return launch(one, std::integral_constant<int, 32>());
    return launch(std::integral_constant<int, 2>(), std::integral_constant<int, 32>());
}

template <typename TL, int CPS>
static AttentionSamples<TL, CPS> attention_samples(const Params& p, const SortParams& sp, uint32_t n) {
    // (a map of K pixels in one row has the most cells)
    const uint32_t K = static_cast<uint32_t>(p.K);
    return {p, sp.fd_p, n, static_cast<uint32_t>(p.P), static_cast<uint32_t>(p.H) * p.LP,
            CPS == 4 ? 2u * (K + 1u) : K, K / static_cast<uint32_t>(p.L)};
}

template <typename T, typename TL>
static cudaError_t launch_sorted_bilinear(const Params& p, SortParams sp,
                                          const LaunchShape& ls, cudaStream_t stream) {
    const uint32_t n = static_cast<uint32_t>(p.Q) * p.P;
    cudaError_t e = launch_sort(attention_samples<TL, 4>(p, sp, n),
                                static_cast<uint32_t>(p.B) * p.H * p.L, sp, ls.sm_count, stream);
    if (e != cudaSuccess) return e;
    auto main = [&](auto nv, auto lpr) {
        constexpr int NV = decltype(nv)::value, LPR = decltype(lpr)::value;
        auto launch = [&](auto kern) { return launch_sorted_main(kern, 32 / LPR, p, sp, n, ls, stream); };
        if (p.D == 4 * NV * LPR) return launch(msda_bwd_sorted_kernel<T, TL, NV, LPR, false, false>);
        if constexpr (NV == 1 && LPR == 32 && sizeof(T) == 2) {   // (see SortedTile)
            const double cells = static_cast<double>(p.B) * p.K * p.H;
            if (sp.nsamples < 40.0 * cells) return launch(msda_bwd_sorted_kernel<T, TL, NV, LPR, true, true>);
        }
        return launch(msda_bwd_sorted_kernel<T, TL, NV, LPR, true, false>);
    };
    return for_row_width(p.D, main);
}

template <typename T>
static cudaError_t launch_sorted_nearest(const Params& p, SortParams sp,
                                         const LaunchShape& ls, cudaStream_t stream) {
    const uint32_t n = static_cast<uint32_t>(p.Q) * p.P;
    cudaError_t e = launch_sort(attention_samples<T, 1>(p, sp, n),
                                static_cast<uint32_t>(p.B) * p.H * p.L, sp, ls.sm_count, stream);
    if (e != cudaSuccess) return e;
    auto main = [&](auto nv, auto lpr) {
        constexpr int NV = decltype(nv)::value, LPR = decltype(lpr)::value;
        return p.D == 4 * NV * LPR
                   ? launch_sorted_main(gka_bwd_sorted_kernel<T, T, NV, LPR, false>, 1, p, sp, n, ls, stream)
                   : launch_sorted_main(gka_bwd_sorted_kernel<T, T, NV, LPR, true>, 1, p, sp, n, ls, stream);
    };
    return for_row_width(p.D, main);
}

}  // namespace msda
