// What the deformable-convolution kernels share: parameters, the position and corners of one
// (pixel, deformable group, tap), channel pieces, and the host's shape checks.
#pragma once

#include <cstdint>

#include "../../include/conv_ops_sm100.h"
#include "msda_launch.h"

namespace dcn {

using msda::FastDiv;
using msda::fd_div;

constexpr int kThreads = 256;

struct DcnParams {
    const float* x;
    const float* offset;
    const float* mask;      // null: not modulated
    float* columns;         // forward: written; backward: grad_columns, read
    float* grad_x;
    float* grad_offset;
    float* grad_mask;
    int H, W, C;
    int Wo, HoWo;
    int K, kw;              // taps, taps per kernel row
    int sh, sw, ph, pw, dh, dw;
    int DG, Cd;             // deformable groups, channels per deformable group
    int Cg, G;              // channels per weight group, weight groups
    int pieces;             // Cd / VEC (VEC = 4 floats per piece, or 1 for odd channel counts)
    int lpi_log2;           // lanes per item = 1 << lpi_log2
    uint32_t items;         // M * DG * K
    FastDiv fd_K, fd_DG, fd_HoWo, fd_Wo, fd_kw, fd_Cg;
};

struct Sample {
    float w[4];        // corner weights (bilinear, times the mask in the forward)
    const float* row[4];  // corner rows of x (this deformable group's channels), null if missing
    float lh, lw;
    bool valid;
};

// Position, corners and weights of item (m, dg, k); every lane of the item's group computes
// the same thing. Fractions come from the fp32 position as in the reference
// (deformable_conv2d.cpp:253-262: floor, then position - floor).
__device__ __forceinline__ void item_setup(const DcnParams& p, uint32_t item, uint32_t* m_out,
                                           uint32_t* dg_out, uint32_t* k_out, float* mask_out,
                                           Sample* s) {
    const uint32_t t = fd_div(item, p.fd_K);
    const uint32_t k = item - t * p.K;
    const uint32_t m = fd_div(t, p.fd_DG);
    const uint32_t dg = t - m * p.DG;
    const uint32_t n = fd_div(m, p.fd_HoWo);
    const uint32_t r = m - n * p.HoWo;
    const uint32_t ho = fd_div(r, p.fd_Wo);
    const uint32_t wo = r - ho * p.Wo;
    const uint32_t ki = fd_div(k, p.fd_kw);
    const uint32_t kj = k - ki * p.kw;
    const float2 d = *reinterpret_cast<const float2*>(
        p.offset + (static_cast<size_t>(m) * p.DG + dg) * (2 * p.K) + 2 * k);
    const float py = static_cast<float>(static_cast<int>(ho) * p.sh - p.ph + static_cast<int>(ki) * p.dh) + d.x;
    const float px = static_cast<float>(static_cast<int>(wo) * p.sw - p.pw + static_cast<int>(kj) * p.dw) + d.y;
    *mask_out = p.mask ? p.mask[(static_cast<size_t>(m) * p.DG + dg) * p.K + k] : 1.f;
    *m_out = m;
    *dg_out = dg;
    *k_out = k;
    const float Hf = static_cast<float>(p.H), Wf = static_cast<float>(p.W);
    s->valid = (py > -1.f) && (px > -1.f) && (py < Hf) && (px < Wf);  // false for NaN
    const float fy = floorf(py), fx = floorf(px);
    const float lh = s->valid ? py - fy : 0.f, lw = s->valid ? px - fx : 0.f;
    const float hh = 1.f - lh, hw = 1.f - lw;
    s->lh = lh;
    s->lw = lw;
    const int y0 = s->valid ? static_cast<int>(fy) : 0, x0 = s->valid ? static_cast<int>(fx) : 0;
    const bool top = y0 >= 0, bottom = y0 + 1 <= p.H - 1, left = x0 >= 0, right = x0 + 1 <= p.W - 1;
    const float* plane = p.x + static_cast<size_t>(n) * p.H * p.W * p.C + static_cast<size_t>(dg) * p.Cd;
    const ptrdiff_t at = (static_cast<ptrdiff_t>(y0) * p.W + x0) * p.C;
    const ptrdiff_t dx = p.C, dy = static_cast<ptrdiff_t>(p.W) * p.C;
    s->row[0] = (s->valid && top && left) ? plane + at : nullptr;
    s->row[1] = (s->valid && top && right) ? plane + at + dx : nullptr;
    s->row[2] = (s->valid && bottom && left) ? plane + at + dy : nullptr;
    s->row[3] = (s->valid && bottom && right) ? plane + at + dy + dx : nullptr;
    s->w[0] = hh * hw;
    s->w[1] = hh * lw;
    s->w[2] = lh * hw;
    s->w[3] = lh * lw;
}

// A piece of a channel row: VEC consecutive floats, kept in a float4 (unused parts zero).
template <int VEC>
__device__ __forceinline__ float4 load_piece(const float* row, int piece) {
    if (row == nullptr) return make_float4(0.f, 0.f, 0.f, 0.f);
    if (VEC == 4) {
        const uint4 r = msda::ldg16(row + 4 * piece);
        return make_float4(__uint_as_float(r.x), __uint_as_float(r.y), __uint_as_float(r.z),
                           __uint_as_float(r.w));
    }
    return make_float4(__ldg(row + piece), 0.f, 0.f, 0.f);
}
template <int VEC>
__device__ __forceinline__ float4 load_column_piece(const float* p) {
    if (VEC == 4) return *reinterpret_cast<const float4*>(p);
    return make_float4(*p, 0.f, 0.f, 0.f);
}
template <int VEC>
__device__ __forceinline__ void store_column_piece(float* p, const float4& v) {
    if (VEC == 4) *reinterpret_cast<float4*>(p) = v;
    else *p = v.x;
}
template <int VEC>
__device__ __forceinline__ void red_piece(float* p, float a, float b, float c, float d) {
    if (VEC == 4) msda::red_add_f32x4(p, a, b, c, d);
    else atomicAdd(p, a);
}

// index of channel c of (m, tap k) in the columns tensor [M, G, K, Cg]
__device__ __forceinline__ size_t column_index(const DcnParams& p, uint32_t m, uint32_t k,
                                               uint32_t c) {
    const uint32_t g = fd_div(c, p.fd_Cg);
    const uint32_t cg = c - g * p.Cg;
    return ((static_cast<size_t>(m) * p.G + g) * p.K + k) * p.Cg + cg;
}

struct Derived {
    long long M;
    int K, Kd, Cg, Cog, Cd;
};

inline int check_shape(const dcn_shape* s, Derived* d) {
    if (s == nullptr) return MSDA_ERR_NULL;
    if (s->N <= 0 || s->H <= 0 || s->W <= 0 || s->C <= 0 || s->Ho <= 0 || s->Wo <= 0 || s->Co <= 0 ||
        s->kh <= 0 || s->kw <= 0 || s->stride_h <= 0 || s->stride_w <= 0 || s->dil_h <= 0 ||
        s->dil_w <= 0 || s->pad_h < 0 || s->pad_w < 0 || s->groups <= 0 || s->deform_groups <= 0)
        return MSDA_ERR_DIMS;
    if (s->C % s->groups != 0 || s->Co % s->groups != 0 || s->C % s->deform_groups != 0)
        return MSDA_ERR_DIMS;
    const int ho = (s->H + 2 * s->pad_h - (s->dil_h * (s->kh - 1) + 1)) / s->stride_h + 1;
    const int wo = (s->W + 2 * s->pad_w - (s->dil_w * (s->kw - 1) + 1)) / s->stride_w + 1;
    if (ho != s->Ho || wo != s->Wo) return MSDA_ERR_DIMS;
    d->M = static_cast<long long>(s->N) * s->Ho * s->Wo;
    d->K = s->kh * s->kw;
    d->Cg = s->C / s->groups;
    d->Cog = s->Co / s->groups;
    d->Cd = s->C / s->deform_groups;
    d->Kd = d->K * d->Cg;
    // 32-bit item and pixel counters in the kernels
    if (d->M * s->deform_groups * d->K >= (1ll << 31) || d->M * s->C * d->K >= (1ll << 40))
        return MSDA_ERR_LIMIT;
    return MSDA_OK;
}

// 16-byte pieces need every row piece and every column piece to start on a 16-byte boundary
inline int piece_width(const dcn_shape* s, const Derived& d) {
    return (d.Cg % 4 == 0 && d.Cd % 4 == 0 && s->C % 4 == 0) ? 4 : 1;
}

inline void fill_params(const dcn_shape* s, const Derived& d, DcnParams* p) {
    p->H = s->H;
    p->W = s->W;
    p->C = s->C;
    p->Wo = s->Wo;
    p->HoWo = s->Ho * s->Wo;
    p->K = d.K;
    p->kw = s->kw;
    p->sh = s->stride_h;
    p->sw = s->stride_w;
    p->ph = s->pad_h;
    p->pw = s->pad_w;
    p->dh = s->dil_h;
    p->dw = s->dil_w;
    p->DG = s->deform_groups;
    p->Cd = d.Cd;
    p->Cg = d.Cg;
    p->G = s->groups;
    p->pieces = d.Cd / piece_width(s, d);
    int l = 0;
    while ((1 << l) < p->pieces && l < 5) ++l;
    p->lpi_log2 = l;
    p->items = static_cast<uint32_t>(d.M * s->deform_groups * d.K);
    p->fd_K = msda::make_fastdiv(d.K);
    p->fd_DG = msda::make_fastdiv(s->deform_groups);
    p->fd_HoWo = msda::make_fastdiv(p->HoWo);
    p->fd_Wo = msda::make_fastdiv(s->Wo);
    p->fd_kw = msda::make_fastdiv(s->kw);
    p->fd_Cg = msda::make_fastdiv(d.Cg);
}

inline size_t round_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// Into how many parts to cut K for a product with few output tiles, so that the persistent
// kernel's CTAs (one per SM) all finish together: the smallest count whose work items fill
// their last round of `sms` to at least 90 %, else the count that fills it best.
inline int balanced_splits(long long tiles, int sms, int max_splits) {
    if (max_splits < 1) max_splits = 1;
    if (max_splits > 64) max_splits = 64;
    int best = 1;
    double best_fill = 0.0;
    for (int s = 1; s <= max_splits; ++s) {
        const long long items = tiles * s;
        const long long rounds = (items + sms - 1) / sms;
        const double fill = static_cast<double>(items) / static_cast<double>(rounds * sms);
        if (fill >= 0.9) return s;
        if (fill > best_fill) {
            best_fill = fill;
            best = s;
        }
    }
    return best;
}

// Parts into which the columns are cut for the forward product: more than one where there are few
// output tiles (small batches), so that every SM has work.
inline int forward_splits(const Derived& d, int sms) {
    const long long tiles = ((d.M + 127) / 128) * static_cast<long long>((d.Cog + 255) / 256);
    return 2 * tiles <= sms ? balanced_splits(tiles, sms, (d.Kd + 255) / 256) : 1;
}

// Parts into which the pixels are cut for the grad_weight product.
inline int weight_splits(const Derived& d, int sms) {
    const long long tiles = ((d.Cog + 127) / 128) * static_cast<long long>((d.Kd + 255) / 256);
    return balanced_splits(tiles, sms, static_cast<int>((d.M + 1023) / 1024));
}

}  // namespace dcn
