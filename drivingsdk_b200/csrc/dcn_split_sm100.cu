// Deformable / modulated deformable convolution from NCHW tensors for sm_100a, products over fp16
// pairs (gemm_split.h). Same decomposition as dcn_sm100.cu (gather, products, scatter), with every
// operand of a product written as pairs by the kernel that produces it:
//   forward   to_nhwc x / offset / mask (and the bounds of x and mask, which bound the columns);
//             weight pairs; gather -> column pairs; out = columns x weight^T
//   backward  bounds and pairs of grad_out, once scaled by pixel (its rows in the product that
//             gives grad_columns) and once by channel (its rows in grad_weight); transposed weight
//             pairs; grad_columns; scatter; grad_weight = grad_out^T x columns
// The column pairs take the bytes that the fp32 columns would. Where x and the mask, or grad_out, spread
// too wide for pairs (range_gate.h) the columns, weights and grad_out are written in fp32 instead, into
// the same memory, and the products over TF32 pairs of dcn_sm100.cu take over; otherwise those return at
// once (some 2 us each).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "../../include/conv_ops_sm100.h"
#include "dcn_common.cuh"
#include "dcn_split.h"
#include "gemm_split.h"
#include "msda_common.cuh"
#include "split_scale.cuh"

namespace {

using namespace dcn;
using msda::SplitOperand;
using msda::SplitScale;
using msda::RangeGate;
using msda::gate_open;
using msda::Elem;

// A tile of a [n][channels][pixels] tensor (or [n][pixels][channels]: channels_last) in shared
// memory as [channel][pixel]; zero outside.
template <typename T, int CH>
__device__ __forceinline__ void load_tile(const T* src, int channels_last, int n, int c0, int p0, int C,
                                          int P, float (&tile)[CH][33]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (!channels_last) {
#pragma unroll
        for (int u = 0; u < CH * 32 / kThreads; ++u) {
            const int r = warp + u * (kThreads / 32);
            const int c = c0 + r, p = p0 + lane;
            tile[r][lane] = (c < C && p < P) ? Elem<T>::to_f(src[(static_cast<size_t>(n) * C + c) * P + p]) : 0.f;
        }
    } else {
#pragma unroll
        for (int u = 0; u < CH * 32 / kThreads; ++u) {
            const int i = warp + u * (kThreads / 32);
            const int r = (i % (CH / 32)) * 32 + lane, q = i / (CH / 32);
            const int c = c0 + r, p = p0 + q;
            tile[r][q] = (c < C && p < P) ? Elem<T>::to_f(src[(static_cast<size_t>(n) * P + p) * C + c]) : 0.f;
        }
    }
    __syncthreads();
}

// Tiles of 32 pixels and some channels of up to three tensors, one CTA each, in one launch: a launch
// costs a small call as much as its work (4 x 128 x 30 x 40 forward and backward: 186 -> 171 us
// for four launches fewer).
struct Tiles {
    uint32_t pixels, channels, count;   // tiles along each, and of the tensor; count 0: no tensor
    FastDiv by_pixels, by_channels;
};
struct Tile {
    int n, c0, p0;
};
Tiles tiles_of(int N, int C, int P, int channels) {
    Tiles t;
    t.pixels = static_cast<uint32_t>((P + 31) / 32);
    t.channels = static_cast<uint32_t>((C + channels - 1) / channels);
    t.count = static_cast<uint32_t>(N) * t.pixels * t.channels;
    t.by_pixels = msda::make_fastdiv(t.pixels);
    t.by_channels = msda::make_fastdiv(t.channels);
    return t;
}
// The tensor and tile of CTA `b`.
template <typename Jobs>
__device__ __forceinline__ int find_tile(const Jobs& jobs, uint32_t b, int channels, Tile& at) {
    int k = 0;
    while (b >= jobs.job[k].tiles.count) b -= jobs.job[k++].tiles.count;
    const Tiles& t = jobs.job[k].tiles;
    const uint32_t row = fd_div(b, t.by_pixels), n = fd_div(row, t.by_channels);
    at.p0 = static_cast<int>(b - row * t.pixels) * 32;
    at.c0 = static_cast<int>(row - n * t.channels) * channels;
    at.n = static_cast<int>(n);
    return k;
}

// Raises *at to v; most callers find it high enough already and skip the atomic.
__device__ __forceinline__ void raise_max(uint32_t* at, uint32_t v) {
    if (v > *reinterpret_cast<volatile uint32_t*>(at)) atomicMax(at, v);
}

// kLeastFrom minus a block's maximum: the larger, the smaller the maximum; 0 for a block of zeros.
__device__ __forceinline__ uint32_t smallness(uint32_t most) { return most == 0u ? 0u : msda::kLeastFrom - most; }

// The same for a tensor's two words of a range (range_gate.h), `which` of two tensors, read together: all
// CTAs of a launch read this one line, which serves about one of them a clock.
__device__ __forceinline__ void raise_range(uint32_t* range, int which, uint32_t most, uint32_t small) {
    uint32_t w[4];
    asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "l"(range) : "memory");
    if (most > (which == 0 ? w[0] : w[1])) atomicMax(range + which, most);
    if (small > (which == 0 ? w[2] : w[3])) atomicMax(range + 2 + which, small);
}

// [n][C][P] (or channels last) in T -> [n][P][C] in fp32; optionally its range, as tensor `which`.
struct LayoutJob {
    Tiles tiles;
    const void* src;
    float* dst;
    int channels_last, C, P;
    uint32_t* range;
    int which;
};
struct LayoutJobs {
    LayoutJob job[3];
};
template <typename T>
__global__ void __launch_bounds__(kThreads)
to_nhwc_kernel(const __grid_constant__ LayoutJobs jobs) {
    __shared__ float tile[32][33];
    Tile at;
    const LayoutJob& job = jobs.job[find_tile(jobs, blockIdx.x, 32, at)];
    const int p0 = at.p0, c0 = at.c0, n = at.n, C = job.C, P = job.P;
    float* __restrict__ dst = job.dst;
    uint32_t* range = job.range;
    const int which = job.which;
    load_tile<T, 32>(static_cast<const T*>(job.src), job.channels_last, n, c0, p0, C, P, tile);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t most = 0, small = 0;   // of this lane's channel; of this warp's pixels
#pragma unroll
    for (int u = 0; u < 1024 / kThreads; ++u) {
        const int r = warp + u * (kThreads / 32);
        const int p = p0 + r, c = c0 + lane;
        const float v = tile[lane][r];
        if (p < P && c < C) dst[(static_cast<size_t>(n) * P + p) * C + c] = v;
        if (range != nullptr) {
            const uint32_t a = msda::finite_magnitude(v);
            most = max(most, a);
            small = max(small, smallness(__reduce_max_sync(0xffffffffu, a)));
        }
    }
    if (range != nullptr) {
        __shared__ uint32_t warp_most[kThreads / 32][32], warp_small[kThreads / 32];
        warp_most[warp][lane] = most;
        if (lane == 0) warp_small[warp] = small;
        __syncthreads();
        if (warp == 0) {
            for (int w = 1; w < kThreads / 32; ++w) {
                most = max(most, warp_most[w][lane]);
                small = max(small, warp_small[w]);
            }
            // single elements are often small: a channel counts with eight pixels or more
            if (P - p0 >= 8) small = max(small, __reduce_max_sync(0xffffffffu, smallness(most)));
            most = __reduce_max_sync(0xffffffffu, most);
            if (lane == 0) raise_range(range, which, most, small);
        }
    }
}

// Rows of a product's operand come from pixel p of image n: n * P + p, or, for weights seen as
// [group][output channel][c * K + k], the column order k * Cg + c.
struct RowOrder {
    int P, K, Cg;   // K == 0: plain
    __device__ __forceinline__ size_t row(int n, int p) const {
        const int q = K == 0 ? p : (p % K) * Cg + p / K;
        return static_cast<size_t>(n) * P + q;
    }
};

// Largest magnitudes of a [n][C][P] tensor per row (pixel) and per channel, and the channel sums;
// optionally its range, over blocks of 64 channels of a pixel.
struct OperandJob {
    Tiles tiles;
    const void* src;
    int channels_last, C;
    RowOrder order;
    uint32_t *row_most, *channel_most;   // channel_most, channel_sum, range: optional
    float* channel_sum;
    uint32_t* range;
    // pairs_kernel: pairs scaled by row, and (optional) scaled by channel or in fp32
    uint16_t *by_row, *by_channel;
    float* plain;
    size_t plane;
    RangeGate if_plain;
};
struct OperandJobs {
    OperandJob job[2];
};
template <typename T>
__global__ void __launch_bounds__(kThreads)
bounds_kernel(const __grid_constant__ OperandJobs jobs) {
    __shared__ float tile[64][33];
    __shared__ uint32_t part[kThreads / 32][32];
    Tile at;
    const OperandJob& job = jobs.job[find_tile(jobs, blockIdx.x, 64, at)];
    const int p0 = at.p0, c0 = at.c0, n = at.n, C = job.C;
    const RowOrder order = job.order;
    uint32_t *row_most = job.row_most, *channel_most = job.channel_most, *range = job.range;
    float* channel_sum = job.channel_sum;
    load_tile<T, 64>(static_cast<const T*>(job.src), job.channels_last, n, c0, p0, C, order.P, tile);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kRows = 64 * 32 / kThreads;    // channels of this warp; lane u keeps the u-th
    uint32_t mine = 0, most = 0;
    float sum = 0.f;
#pragma unroll
    for (int u = 0; u < kRows; ++u) {
        const float v = tile[warp + u * (kThreads / 32)][lane];
        const uint32_t a = msda::finite_magnitude(v);
        mine = max(mine, a);
        if (channel_most != nullptr) {
            const uint32_t m = __reduce_max_sync(0xffffffffu, a);
            if (lane == u) most = m;
        }
        if (channel_sum != nullptr) {
            float s = v;
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == u) sum = s;
        }
    }
    const int channel = c0 + warp + lane * (kThreads / 32);
    if (lane < kRows && channel < C) {
        if (channel_most != nullptr) raise_max(channel_most + channel, most);
        if (channel_sum != nullptr) atomicAdd(channel_sum + channel, sum);
    }
    part[warp][lane] = mine;
    __syncthreads();
    if (warp == 0) {
        for (int w = 1; w < kThreads / 32; ++w) mine = max(mine, part[w][lane]);
        if (p0 + lane < order.P) raise_max(row_most + order.row(n, p0 + lane), mine);
        if (range != nullptr) {
            const uint32_t small = __reduce_max_sync(0xffffffffu, smallness(mine));
            const uint32_t tile_most = __reduce_max_sync(0xffffffffu, mine);
            if (lane == 0) raise_range(range, 0, tile_most, small);
        }
    }
}

// [n][C][P] -> pairs [rows][C] scaled by row, and (optional) the same scaled by channel or in fp32:
// where both are given, in fp32 if the gate is open.
template <typename T>
__global__ void __launch_bounds__(kThreads)
pairs_kernel(const __grid_constant__ OperandJobs jobs) {
    __shared__ float tile[64][33];
    Tile tile_at;
    const OperandJob& job = jobs.job[find_tile(jobs, blockIdx.x, 64, tile_at)];
    const int p0 = tile_at.p0, c0 = tile_at.c0, n = tile_at.n, C = job.C;
    const RowOrder order = job.order;
    const uint32_t *row_most = job.row_most, *channel_most = job.channel_most;
    uint16_t *by_row = job.by_row, *by_channel = job.by_channel;
    float* plain = job.plain;
    const size_t plane = job.plane;
    if (by_channel != nullptr && plain != nullptr) {
        if (gate_open(job.if_plain)) by_channel = nullptr;
        else plain = nullptr;
    }
    load_tile<T, 64>(static_cast<const T*>(job.src), job.channels_last, n, c0, p0, C, order.P, tile);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c = c0 + 2 * lane;
    if (c >= C) return;   // C is even
    float sc[2] = {1.f, 1.f};
    if (by_channel != nullptr) {
        sc[0] = msda::exp2_int(msda::split_exponent(SplitScale{channel_most, 1, nullptr}, c));
        sc[1] = msda::exp2_int(msda::split_exponent(SplitScale{channel_most, 1, nullptr}, c + 1));
    }
#pragma unroll
    for (int q = warp; q < 32; q += kThreads / 32) {
        if (p0 + q >= order.P) break;
        const size_t row = order.row(n, p0 + q);
        const float x = tile[2 * lane][q], y = tile[2 * lane + 1][q];
        const float sr = msda::exp2_int(msda::split_exponent(SplitScale{row_most, 1, nullptr}, row));
        const uint2 r = msda::split_pair(x, y, sr);
        uint16_t* at = by_row + row * C + c;
        *reinterpret_cast<uint32_t*>(at) = r.x;
        *reinterpret_cast<uint32_t*>(at + plane) = r.y;
        if (plain != nullptr) *reinterpret_cast<float2*>(plain + row * C + c) = make_float2(x, y);
        if (by_channel != nullptr) {
            const uint2 h = msda::split_pair(x * sc[0], y * sc[1], 1.f);
            uint16_t* to = by_channel + row * C + c;
            *reinterpret_cast<uint32_t*>(to) = h.x;
            *reinterpret_cast<uint32_t*>(to + plane) = h.y;
        }
    }
}

// weight [Co][Cg][K] -> pairs [Co][K * Cg], one CTA per output channel, scaled by it; or in fp32, into
// the same memory, where the columns' range is wide.
template <typename T>
__global__ void __launch_bounds__(kThreads)
weight_pairs_kernel(const T* __restrict__ w, int Cg, int K, uint32_t* most, uint16_t* __restrict__ pairs,
                    size_t plane, const uint32_t* columns_range) {
    __shared__ uint32_t warp_most[kThreads / 32];
    const int co = blockIdx.x, Kd = Cg * K;
    const T* src = w + static_cast<size_t>(co) * Kd;
    if (msda::range_is_wide(columns_range)) {
        float* to = reinterpret_cast<float*>(pairs) + static_cast<size_t>(co) * Kd;
        for (int i = threadIdx.x; i < Kd; i += kThreads) {
            const int k = i / Cg, c = i - k * Cg;
            to[i] = Elem<T>::to_f(src[c * K + k]);
        }
        return;
    }
    uint32_t m = 0;
    for (int i = threadIdx.x; i < Kd; i += kThreads) m = max(m, msda::finite_magnitude(Elem<T>::to_f(src[i])));
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) warp_most[threadIdx.x >> 5] = m;
    __syncthreads();
    for (int i = 0; i < kThreads / 32; ++i) m = max(m, warp_most[i]);
    if (threadIdx.x == 0) most[co] = m;
    const uint32_t bound = m;
    const float s = msda::exp2_int(msda::split_exponent(SplitScale{&bound, 0, nullptr}, 0));
    for (int i = threadIdx.x; i < Kd / 2; i += kThreads) {
        const int at = 2 * i, k = at / Cg, c = at - k * Cg;   // Cg is even
        const uint2 r = msda::split_pair(Elem<T>::to_f(src[c * K + k]), Elem<T>::to_f(src[(c + 1) * K + k]), s);
        uint16_t* to = pairs + static_cast<size_t>(co) * Kd + at;
        *reinterpret_cast<uint32_t*>(to) = r.x;
        *reinterpret_cast<uint32_t*>(to + plane) = r.y;
    }
}

// Column pairs: mask * bilinear(x), pixel by pixel. A group of lanes per (pixel, deformable group, tap)
// moves pieces of eight channels.
__global__ void __launch_bounds__(kThreads, 4)
gather_pairs_kernel(const __grid_constant__ DcnParams p, const __grid_constant__ ColumnsOut out) {
    const int lpi = 1 << p.lpi_log2;
    const int sub = threadIdx.x & (lpi - 1);
    const uint32_t slot = threadIdx.x >> p.lpi_log2;             // item within the CTA's step
    const uint32_t per_step = static_cast<uint32_t>(kThreads) >> p.lpi_log2;
    const float scale = msda::exp2_int(msda::split_exponent(out.bound, 0));
    const bool pairs = !msda::range_is_wide(out.range), plain = !pairs || out.keep_f32;
#pragma unroll 1
    for (uint32_t item = blockIdx.x * per_step + slot; item < p.items; item += gridDim.x * per_step) {
        uint32_t m, dg, k;
        float mk;
        Sample s;
        item_setup(p, item, &m, &dg, &k, &mk, &s);
        for (int piece = sub; piece < p.pieces; piece += lpi) {
            float4 acc[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
            if (s.valid) {
                float4 v[4][2];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    v[c][0] = load_piece<4>(s.row[c], 2 * piece);
                    v[c][1] = load_piece<4>(s.row[c], 2 * piece + 1);
                }
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float w = s.w[c] * mk;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        acc[h].x = fmaf(w, v[c][h].x, acc[h].x);
                        acc[h].y = fmaf(w, v[c][h].y, acc[h].y);
                        acc[h].z = fmaf(w, v[c][h].z, acc[h].z);
                        acc[h].w = fmaf(w, v[c][h].w, acc[h].w);
                    }
                }
            }
            const size_t to_at = column_index(p, m, k, dg * p.Cd + 8 * piece);
            if (plain) {
                *reinterpret_cast<float4*>(out.f32 + to_at) = acc[0];
                *reinterpret_cast<float4*>(out.f32 + to_at + 4) = acc[1];
            }
            if (pairs) {
                const uint2 r0 = msda::split_pair(acc[0].x, acc[0].y, scale);
                const uint2 r1 = msda::split_pair(acc[0].z, acc[0].w, scale);
                const uint2 r2 = msda::split_pair(acc[1].x, acc[1].y, scale);
                const uint2 r3 = msda::split_pair(acc[1].z, acc[1].w, scale);
                uint16_t* to = out.pairs + to_at;
                *reinterpret_cast<uint4*>(to) = make_uint4(r0.x, r1.x, r2.x, r3.x);
                *reinterpret_cast<uint4*>(to + out.plane) = make_uint4(r0.y, r1.y, r2.y, r3.y);
            }
        }
    }
}

// The columns as grad_weight's fp32 product wants them, from what the forward saved: pairs put together
// again (22 bits, and narrow, or they would be fp32), or the fp32 columns.
__global__ void __launch_bounds__(kThreads)
join_columns_kernel(const void* __restrict__ saved, const uint32_t* columns_range, SplitScale bound, size_t plane,
                    float* __restrict__ out, const RangeGate gate) {
    if (!gate_open(gate)) return;
    const bool f32 = msda::range_is_wide(columns_range);
    const float back = msda::exp2_int(-msda::split_exponent(bound, 0));
    const size_t step = static_cast<size_t>(gridDim.x) * kThreads * 4;
    for (size_t i = (static_cast<size_t>(blockIdx.x) * kThreads + threadIdx.x) * 4; i < plane; i += step) {
        float4 v;
        if (f32) {
            v = *reinterpret_cast<const float4*>(static_cast<const float*>(saved) + i);
        } else {
            const __half* hi = static_cast<const __half*>(saved) + i;
            float sum[4];
            for (int e = 0; e < 4; ++e) sum[e] = (__half2float(hi[e]) + __half2float(hi[plane + e])) * back;
            v = make_float4(sum[0], sum[1], sum[2], sum[3]);
        }
        *reinterpret_cast<float4*>(out + i) = v;
    }
}

size_t up(size_t v) { return (v + 255) / 256 * 256; }

// Sampling over cell-sorted samples instead of pixel by pixel: pays where rows are long enough to
// occupy a warp and the sort (some 15 us at least) is small against the sampling. Forward and backward,
// pixel by pixel / sorted, in us: Cd = 512, 235 k samples 1510 / 1265; Cd = 128, 0.69 M 1445 / 1055,
// 0.17 M 369 / 290, 43 k 170 / 174; Cd = 64, 0.17 M 241 / 233 but 67 / 79 for the forward alone,
// Cd = 16, 0.69 M 251 / 356.
bool sort_pays(const dcn_shape* s, const Derived& d) {
    return d.Cd >= 96 && d.M * s->deform_groups * d.K >= 100000 && dcn::sorted_bytes(s, d) != 0;
}

// Whether grad_weight is formed from fp32 operands by the TF32 kernel whatever their range. The tensor
// core truncates as it accumulates, so a sum's error grows with its chain of products: at 13050 pixels
// a chain the TF32 sums are 9.2e-5 of the result off float64, the pair sums 4.7e-5 off the TF32 sums.
// The two forms of this operator (the extension's own entry points use the other) are held to agree to
// 2e-5 for fp32 tensors: past 4000 pixels a chain, where the distance by that measurement would reach
// 1.4e-5, this one uses the other's kernel (508 us instead of 258 at 26100 x 512 x 4608).
bool weight_in_f32(const Derived& d, int dtype) {
    int sms = 148;
    msda::device_facts(&sms, nullptr);
    return dtype == MSDA_F32 && d.M > 4000ll * weight_splits(d, sms);
}

// What the forward leaves for the backward: bounds, x, offset and mask as [n][pixel][channel] fp32,
// the samples in cell order, and the columns as grad_weight wants them. `keep` == 0: no backward
// will follow. The pairs of the columns are there too, or in the forward's workspace.
struct Saved {
    size_t bounds, x, offset, mask, sorted, columns, total;
    size_t plane;   // halves per plane of the columns
    bool f32;       // columns in fp32 (else pairs, or fp32 where their range is wide)
};
Saved plan_saved(const dcn_shape* s, const Derived& d, int dtype, bool keep) {
    Saved r;
    r.bounds = 0;
    r.x = 256;
    r.offset = r.x + up(static_cast<size_t>(s->N) * s->H * s->W * s->C * 4);
    const size_t taps = static_cast<size_t>(d.M) * s->deform_groups * d.K;
    r.mask = r.offset + up(taps * 8);
    r.sorted = r.mask + up(taps * 4);
    r.columns = r.sorted + up(sort_pays(s, d) ? dcn::sorted_bytes(s, d) : 0);
    r.plane = static_cast<size_t>(d.M) * s->groups * d.Kd;
    r.total = r.columns + up(r.plane * 4) + 256;   // row blocks of 64 may be read past the end
    r.f32 = keep && weight_in_f32(d, dtype);
    return r;
}

struct BackwardSpace {
    size_t ticket, go_range, grad_columns, go_rows, go_channels, weight_t, row_most, channel_most, weight_most, total;
};
BackwardSpace plan_backward(const dcn_shape* s, const Derived& d) {
    BackwardSpace r;
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t here = at;
        at += up(bytes);
        return here;
    };
    const size_t go = static_cast<size_t>(d.M) * s->Co;
    const size_t rows = static_cast<size_t>(s->groups) * d.Kd;
    r.ticket = take(sizeof(uint32_t));                     // these five: cleared together
    r.go_range = take(4 * sizeof(uint32_t));
    r.row_most = take(static_cast<size_t>(d.M) * 4);
    r.channel_most = take(static_cast<size_t>(s->Co) * 4);
    r.weight_most = take(rows * 4);
    r.grad_columns = take(static_cast<size_t>(d.M) * rows * 4);
    r.go_rows = take(go * 4);
    r.go_channels = take(go * 4 + 256);
    r.weight_t = take(rows * d.Cog * 4);
    r.total = at;
    return r;
}

struct ForwardSpace {
    size_t weight_most, weight, columns, total;
};
ForwardSpace plan_forward(const dcn_shape* s, const Derived& d, const Saved& at) {
    ForwardSpace r;
    r.weight_most = 0;
    r.weight = up(static_cast<size_t>(s->Co) * 4);
    r.columns = r.weight + up(static_cast<size_t>(s->Co) * d.Kd * 4);
    r.total = r.columns + (at.f32 ? up(at.plane * 4) : 0);
    return r;
}

#define RETURN_ON_CUDA(expr)                                          \
    do {                                                              \
        const cudaError_t err_ = (expr);                              \
        if (err_ != cudaSuccess) return msda::note_cuda_error(err_);  \
    } while (0)

void sample_params(const dcn_shape* s, const Derived& d, const char* saved, const Saved& at, bool masked,
                   DcnParams* p) {
    fill_params(s, d, p);
    p->x = reinterpret_cast<const float*>(saved + at.x);
    p->offset = reinterpret_cast<const float*>(saved + at.offset);
    p->mask = masked ? reinterpret_cast<const float*>(saved + at.mask) : nullptr;
}

template <typename T>
int forward_typed(const void* x, int x_nhwc, const void* offset, const void* mask, const void* weight,
                  const float* bias, float* out, char* saved, char* ws, const dcn_shape* s, const Derived& d,
                  const Saved& at, cudaStream_t stream) {
    int sms = 0;
    int* status = nullptr;
    int rc = msda::device_facts(&sms, &status);
    if (rc != MSDA_OK) return rc;
    const ForwardSpace sp = plan_forward(s, d, at);
    uint32_t* bounds = reinterpret_cast<uint32_t*>(saved + at.bounds);
    RETURN_ON_CUDA(cudaMemsetAsync(bounds, 0, 16, stream));
    const int HoWo = s->Ho * s->Wo, taps = s->deform_groups * d.K;
    auto place = [&](size_t offset_in_saved) { return reinterpret_cast<float*>(saved + offset_in_saved); };
    const LayoutJobs jobs{{{tiles_of(s->N, s->C, s->H * s->W, 32), x, place(at.x), x_nhwc, s->C, s->H * s->W, bounds,
                            0},
                           {tiles_of(s->N, 2 * taps, HoWo, 32), offset, place(at.offset), 0, 2 * taps, HoWo, nullptr,
                            0},
                           {tiles_of(mask != nullptr ? s->N : 0, taps, HoWo, 32), mask, place(at.mask), 0, taps, HoWo,
                            bounds, 1}}};
    to_nhwc_kernel<T><<<jobs.job[0].tiles.count + jobs.job[1].tiles.count + jobs.job[2].tiles.count, kThreads, 0,
                        stream>>>(jobs);
    RETURN_ON_CUDA(cudaGetLastError());
    msda::count_launches(1);
    const size_t wplane = static_cast<size_t>(s->Co) * d.Kd;
    uint16_t* wpairs = reinterpret_cast<uint16_t*>(ws + sp.weight);
    uint32_t* wmost = reinterpret_cast<uint32_t*>(ws + sp.weight_most);
    weight_pairs_kernel<T><<<s->Co, kThreads, 0, stream>>>(static_cast<const T*>(weight), d.Cg, d.K, wmost,
                                                          wpairs, wplane, bounds);
    RETURN_ON_CUDA(cudaGetLastError());

    DcnParams p{};
    sample_params(s, d, saved, at, mask != nullptr, &p);
    uint16_t* columns = reinterpret_cast<uint16_t*>(at.f32 ? ws + sp.columns : saved + at.columns);
    float* columns_f32 = reinterpret_cast<float*>(saved + at.columns);
    const SplitScale col_scale{bounds, 0, mask != nullptr ? bounds + 1 : nullptr};
    const ColumnsOut to{columns, at.plane, columns_f32, at.f32 ? 1 : 0, col_scale, bounds};
    msda::count_launches(1);
    if (sort_pays(s, d)) {
        rc = launch_gather_sorted(p, saved + at.sorted, d.M, s->N, to, sms, stream);
        if (rc != MSDA_OK) return rc;
    } else {
        p.pieces = d.Cd / 8;
        int l = 0;
        while ((1 << l) < p.pieces && l < 5) ++l;
        p.lpi_log2 = l;
        int per_sm = 0;
        RETURN_ON_CUDA(msda::resident_ctas(reinterpret_cast<const void*>(gather_pairs_kernel), kThreads, 0, &per_sm));
        const uint32_t per_step = static_cast<uint32_t>(kThreads) >> p.lpi_log2;
        const uint32_t want = (p.items + per_step - 1) / per_step, cap = static_cast<uint32_t>(sms) * per_sm;
        gather_pairs_kernel<<<want < cap ? want : cap, kThreads, 0, stream>>>(p, to);
        RETURN_ON_CUDA(cudaGetLastError());
        msda::count_launches(1);
    }

    const int splits = forward_splits(d, sms);
    if (splits > 1) RETURN_ON_CUDA(cudaMemsetAsync(out, 0, static_cast<size_t>(d.M) * s->Co * 4, stream));
    for (int g = 0; g < s->groups; ++g) {
        const SplitOperand A{columns + static_cast<size_t>(g) * d.Kd, static_cast<long long>(s->groups) * d.Kd, 1,
                             static_cast<long long>(at.plane), col_scale};
        const SplitOperand B{wpairs + static_cast<size_t>(g) * d.Cog * d.Kd, d.Kd, 1,
                             static_cast<long long>(wplane), SplitScale{wmost + g * d.Cog, 1, nullptr}};
        RETURN_ON_CUDA(msda::gemm_split(A, B, out + static_cast<size_t>(g) * d.Cog, s->Co,
                                        bias != nullptr ? bias + g * d.Cog : nullptr, static_cast<int>(d.M),
                                        d.Cog, d.Kd, splits, RangeGate{{bounds, nullptr}, 0}, status, stream));
        msda::count_launches(1);
    }
    return launch_forward_product(columns_f32, reinterpret_cast<const float*>(wpairs), bias, out, s, d, sms,
                                  RangeGate{{bounds, nullptr}, 1}, status, stream);
}

template <typename T>
int backward_typed(const void* weight, const void* grad_out, int go_nhwc, const char* saved, bool masked,
                   float* grad_x, float* grad_offset, float* grad_mask, float* grad_weight, float* grad_bias,
                   char* ws, const dcn_shape* s, const Derived& d, const Saved& at, cudaStream_t stream) {
    int sms = 0;
    int* status = nullptr;
    int rc = msda::device_facts(&sms, &status);
    if (rc != MSDA_OK) return rc;
    const bool weight_f32 = at.f32;
    const BackwardSpace sp = plan_backward(s, d);
    const int M = static_cast<int>(d.M), HoWo = s->Ho * s->Wo;
    const uint32_t* bounds = reinterpret_cast<const uint32_t*>(saved + at.bounds);
    uint32_t* row_most = reinterpret_cast<uint32_t*>(ws + sp.row_most);
    uint32_t* channel_most = reinterpret_cast<uint32_t*>(ws + sp.channel_most);
    uint32_t* weight_most = reinterpret_cast<uint32_t*>(ws + sp.weight_most);
    uint16_t* go_rows = reinterpret_cast<uint16_t*>(ws + sp.go_rows);
    uint16_t* go_channels = reinterpret_cast<uint16_t*>(ws + sp.go_channels);
    uint16_t* weight_t = reinterpret_cast<uint16_t*>(ws + sp.weight_t);
    float* grad_columns = reinterpret_cast<float*>(ws + sp.grad_columns);
    uint32_t* go_range = reinterpret_cast<uint32_t*>(ws + sp.go_range);
    const RangeGate narrow{{bounds, go_range}, 0}, wide{{bounds, go_range}, 1};
    RETURN_ON_CUDA(cudaMemsetAsync(ws + sp.ticket, 0, sp.grad_columns - sp.ticket, stream));
    if (grad_bias != nullptr) RETURN_ON_CUDA(cudaMemsetAsync(grad_bias, 0, static_cast<size_t>(s->Co) * 4, stream));
    RETURN_ON_CUDA(cudaMemsetAsync(grad_x, 0, static_cast<size_t>(s->N) * s->H * s->W * s->C * 4, stream));

    // grad_out, and the weights as [group][kd][output channel]: bounds, then pairs (the second reading
    // mostly comes from L2)
    const size_t go_plane = static_cast<size_t>(M) * s->Co;
    const size_t wt_plane = static_cast<size_t>(s->groups) * d.Kd * d.Cog;
    {
        OperandJobs jobs{};
        OperandJob &go = jobs.job[0], &w = jobs.job[1];
        go.tiles = tiles_of(s->N, s->Co, HoWo, 64);
        go.src = grad_out;
        go.channels_last = go_nhwc;
        go.C = s->Co;
        go.order = RowOrder{HoWo, 0, 0};
        go.row_most = row_most;
        go.channel_most = channel_most;
        go.channel_sum = grad_bias;
        go.range = go_range;
        go.by_row = go_rows;
        go.by_channel = weight_f32 ? nullptr : go_channels;
        go.plain = reinterpret_cast<float*>(go_channels);
        go.plane = go_plane;
        go.if_plain = wide;
        w.tiles = tiles_of(s->groups, d.Cog, d.Kd, 64);
        w.src = weight;
        w.C = d.Cog;
        w.order = RowOrder{d.Kd, d.K, d.Cg};
        w.row_most = weight_most;
        w.by_row = weight_t;
        w.plane = wt_plane;
        const uint32_t grid = go.tiles.count + w.tiles.count;
        bounds_kernel<T><<<grid, kThreads, 0, stream>>>(jobs);
        pairs_kernel<T><<<grid, kThreads, 0, stream>>>(jobs);
    }
    RETURN_ON_CUDA(cudaGetLastError());
    msda::count_launches(2);

    const long long ld_cols = static_cast<long long>(s->groups) * d.Kd;
    for (int g = 0; g < s->groups; ++g) {
        const SplitOperand A{go_rows + static_cast<size_t>(g) * d.Cog, s->Co, 1, static_cast<long long>(go_plane),
                             SplitScale{row_most, 1, nullptr}};
        const SplitOperand B{weight_t + static_cast<size_t>(g) * d.Kd * d.Cog, d.Cog, 1,
                             static_cast<long long>(wt_plane),
                             SplitScale{weight_most + static_cast<size_t>(g) * d.Kd, 1, nullptr}};
        RETURN_ON_CUDA(msda::gemm_split(A, B, grad_columns + static_cast<size_t>(g) * d.Kd, ld_cols, nullptr, M,
                                        d.Kd, d.Cog, 1, RangeGate{}, status, stream));
        msda::count_launches(1);
    }

    DcnParams p{};
    sample_params(s, d, saved, at, masked, &p);
    p.columns = grad_columns;
    p.grad_x = grad_x;
    p.grad_offset = grad_offset;
    p.grad_mask = grad_mask;
    if (sort_pays(s, d))
        rc = launch_scatter_sorted(p, saved + at.sorted, reinterpret_cast<uint32_t*>(ws + sp.ticket), d.M, s->N, sms,
                                   stream);
    else rc = launch_scatter(p, sms, stream);
    if (rc != MSDA_OK) return rc;

    if (weight_f32)
        return launch_weight_product(reinterpret_cast<const float*>(go_channels),
                                     reinterpret_cast<const float*>(saved + at.columns), grad_weight, s, d, sms,
                                     RangeGate{}, status, stream);
    const uint16_t* columns = reinterpret_cast<const uint16_t*>(saved + at.columns);
    const SplitScale col_scale{bounds, 0, masked ? bounds + 1 : nullptr};
    const int splits = weight_splits(d, sms);
    if (splits > 1)
        RETURN_ON_CUDA(cudaMemsetAsync(grad_weight, 0, static_cast<size_t>(s->Co) * d.Kd * 4, stream));
    for (int g = 0; g < s->groups; ++g) {
        const SplitOperand A{go_channels + static_cast<size_t>(g) * d.Cog, 1, s->Co, static_cast<long long>(go_plane),
                             SplitScale{channel_most + static_cast<size_t>(g) * d.Cog, 1, nullptr}};
        const SplitOperand B{columns + static_cast<size_t>(g) * d.Kd, 1, ld_cols, static_cast<long long>(at.plane),
                             col_scale};
        RETURN_ON_CUDA(msda::gemm_split(A, B, grad_weight + static_cast<size_t>(g) * d.Cog * d.Kd, d.Kd, nullptr,
                                        d.Cog, d.Kd, M, splits, narrow, status, stream));
        msda::count_launches(1);
    }
    // or, where a range is wide, over the fp32 columns (the gradient of the columns is used up)
    join_columns_kernel<<<2 * sms, kThreads, 0, stream>>>(columns, bounds, col_scale, at.plane, grad_columns, wide);
    RETURN_ON_CUDA(cudaGetLastError());
    msda::count_launches(1);
    return launch_weight_product(reinterpret_cast<const float*>(go_channels), grad_columns, grad_weight, s, d, sms,
                                 wide, status, stream);
}

int split_shape(const dcn_shape* s, Derived* d) {
    const int rc = check_shape(s, d);
    if (rc != MSDA_OK) return rc;
    // 16-byte pieces of halves in every row
    if (d->Cg % 8 != 0 || d->Cd % 8 != 0 || d->Cog % 8 != 0) return MSDA_ERR_ALIGN;
    // one CTA per tile in the layout kernels
    const long long HoWo = static_cast<long long>(s->Ho) * s->Wo, taps = static_cast<long long>(s->deform_groups) * d->K;
    auto tiles = [](long long n, long long C, long long P) { return n * ((C + 31) / 32) * ((P + 31) / 32); };
    const long long most = tiles(s->N, s->C, static_cast<long long>(s->H) * s->W) + tiles(s->N, 3 * taps, HoWo) + s->N +
                           tiles(s->N, s->Co, HoWo) + tiles(s->groups, d->Cog, d->Kd);
    return most < (1ll << 31) ? MSDA_OK : MSDA_ERR_LIMIT;
}

}  // namespace

extern "C" {

size_t dcn_sm100_saved_bytes(const dcn_shape* s, int dtype, int keep) {
    Derived d;
    return split_shape(s, &d) == MSDA_OK && dcn_sm100_use_tensor_cores(-1) == 1
               ? plan_saved(s, d, dtype, keep != 0).total : 0;
}

size_t dcn_sm100_nchw_workspace_bytes(const dcn_shape* s, int dtype, int keep, int backward) {
    Derived d;
    if (check_shape(s, &d) != MSDA_OK) return 0;
    return backward ? plan_backward(s, d).total : plan_forward(s, d, plan_saved(s, d, dtype, keep != 0)).total;
}

int dcn_sm100_forward_nchw(const void* x, int x_nhwc, const void* offset, const void* mask, const void* weight,
                           const float* bias, float* out, void* saved, size_t saved_bytes, void* workspace,
                           size_t workspace_bytes, const dcn_shape* s, int dtype, int keep, void* stream_v) {
    if (x == nullptr || offset == nullptr || weight == nullptr || out == nullptr || saved == nullptr ||
        workspace == nullptr)
        return MSDA_ERR_NULL;
    Derived d;
    const int rc = split_shape(s, &d);
    if (rc != MSDA_OK) return rc;
    if (dcn_sm100_use_tensor_cores(-1) != 1) return MSDA_ERR_LIMIT;
    const Saved at = plan_saved(s, d, dtype, keep != 0);
    if (saved_bytes < at.total || workspace_bytes < plan_forward(s, d, at).total)
        return MSDA_ERR_WORKSPACE;
    if ((reinterpret_cast<uintptr_t>(saved) | reinterpret_cast<uintptr_t>(workspace)) % 16 != 0) return MSDA_ERR_ALIGN;
    char* sv = static_cast<char*>(saved);
    char* ws = static_cast<char*>(workspace);
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    switch (dtype) {
        case MSDA_F32: return forward_typed<float>(x, x_nhwc, offset, mask, weight, bias, out, sv, ws, s, d, at, stream);
        case MSDA_F16: return forward_typed<__half>(x, x_nhwc, offset, mask, weight, bias, out, sv, ws, s, d, at, stream);
        case MSDA_BF16:
            return forward_typed<__nv_bfloat16>(x, x_nhwc, offset, mask, weight, bias, out, sv, ws, s, d, at, stream);
        default: return MSDA_ERR_DTYPE;
    }
}

int dcn_sm100_backward_nchw(const void* weight, const void* grad_out, int grad_out_nhwc, const void* saved,
                            float* grad_x, float* grad_offset, float* grad_mask, float* grad_weight,
                            float* grad_bias, void* workspace, size_t workspace_bytes, const dcn_shape* s,
                            int dtype, void* stream_v) {
    if (weight == nullptr || grad_out == nullptr || saved == nullptr || grad_x == nullptr ||
        grad_offset == nullptr || grad_weight == nullptr || workspace == nullptr)
        return MSDA_ERR_NULL;
    Derived d;
    const int rc = split_shape(s, &d);
    if (rc != MSDA_OK) return rc;
    if (workspace_bytes < plan_backward(s, d).total) return MSDA_ERR_WORKSPACE;
    if ((reinterpret_cast<uintptr_t>(saved) | reinterpret_cast<uintptr_t>(workspace) |
         reinterpret_cast<uintptr_t>(grad_x)) % 16 != 0 || reinterpret_cast<uintptr_t>(grad_offset) % 8 != 0)
        return MSDA_ERR_ALIGN;
    const char* sv = static_cast<const char*>(saved);
    char* ws = static_cast<char*>(workspace);
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    const bool masked = grad_mask != nullptr;
    const Saved at = plan_saved(s, d, dtype, true);
    switch (dtype) {
        case MSDA_F32:
            return backward_typed<float>(weight, grad_out, grad_out_nhwc, sv, masked, grad_x, grad_offset,
                                         grad_mask, grad_weight, grad_bias, ws, s, d, at, stream);
        case MSDA_F16:
            return backward_typed<__half>(weight, grad_out, grad_out_nhwc, sv, masked, grad_x, grad_offset,
                                          grad_mask, grad_weight, grad_bias, ws, s, d, at, stream);
        case MSDA_BF16:
            return backward_typed<__nv_bfloat16>(weight, grad_out, grad_out_nhwc, sv, masked, grad_x,
                                                 grad_offset, grad_mask, grad_weight, grad_bias, ws, s, d, at, stream);
        default: return MSDA_ERR_DTYPE;
    }
}

}  // extern "C"
