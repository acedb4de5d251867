// C-ABI entry points of the sm_100a MSDA library: argument validation, the
// launch plan (what the reference computes in its host tiling functions,
// kernels/multi_scale_deformable_attn/op_host/multi_scale_deformable_attn.cpp:32-114
// and multi_scale_deformable_attn_grad.cpp:35-86), and kernel launches.
// No allocation, no synchronisation (except msda_sm100_device_status).
#include <atomic>
#include <cmath>
#include <cstring>

#include "../../include/msda_sm100.h"
#include "msda_launch.h"
#include "sort_plan.h"

namespace {

using msda::Params;
using msda::RowPlan;

constexpr int kAbiVersion = 1;
constexpr int kBilinear = 0, kNearest = 1, kFused = 2;
constexpr int kMaxDevices = 64;

__device__ int g_status_word;

std::atomic<int> g_tune_stage{2};   // 0 never, 1 both directions, 2 backward kernels only
std::atomic<int> g_tune_interleave{1};
std::atomic<int> g_tune_cps_fwd{0};
std::atomic<int> g_tune_cps_bwd{0};
std::atomic<int> g_tune_spin{msda::kSpinLimit};
std::atomic<int> g_tune_precise_amp{8};
std::atomic<int> g_tune_debug_rows{0};
std::atomic<int> g_tune_pack{1};
std::atomic<int> g_tune_sort{1};
std::atomic<long long> g_launches{0};
thread_local int t_last_cuda_error = 0;
thread_local cudaEvent_t t_prof[4] = {nullptr, nullptr, nullptr, nullptr};

void prof_record(int which, cudaStream_t stream) {
    if (t_prof[which] != nullptr) cudaEventRecord(t_prof[which], stream);
}

struct DeviceInfo {
    std::atomic<int> ready{0};
    int sm_count = 0;
    int* status_ptr = nullptr;
};
DeviceInfo g_dev[kMaxDevices];

int fail_cuda(cudaError_t e) {
    t_last_cuda_error = static_cast<int>(e);
    return MSDA_ERR_CUDA;
}

// Per-device facts (SM count, address of the status word), looked up once.
// Racing first calls do the same idempotent work.
int device_info(const DeviceInfo** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail_cuda(e);
    if (dev < 0 || dev >= kMaxDevices) return MSDA_ERR_LIMIT;
    DeviceInfo& d = g_dev[dev];
    if (!d.ready.load(std::memory_order_acquire)) {
        int sms = 0;
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return fail_cuda(e);
        void* sp = nullptr;
        e = cudaGetSymbolAddress(&sp, g_status_word);
        if (e != cudaSuccess) return fail_cuda(e);
        d.sm_count = sms;
        d.status_ptr = static_cast<int*>(sp);
        d.ready.store(1, std::memory_order_release);
    }
    *out = &d;
    return MSDA_OK;
}

size_t elem_size(int dtype) { return dtype == MSDA_F32 ? 4 : 2; }

bool aligned_to(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

// Is this pointer device-accessible memory (device or managed)? Unregistered
// host memory reports cudaMemoryTypeUnregistered.
int pointer_on_device(const void* p, bool* on_device) {
    cudaPointerAttributes attr;
    cudaError_t e = cudaPointerGetAttributes(&attr, p);
    if (e != cudaSuccess) {
        cudaGetLastError();
        *on_device = false;
        return MSDA_OK;
    }
    *on_device = (attr.type == cudaMemoryTypeDevice || attr.type == cudaMemoryTypeManaged);
    return MSDA_OK;
}

// Separates the level-table flags from a dtype argument.
int split_flags(int* dtype) {
    const int flags = *dtype & (MSDA_TABLES_INT64 | MSDA_TABLES_DEVICE);
    if (*dtype >= 0) *dtype &= ~(MSDA_TABLES_INT64 | MSDA_TABLES_DEVICE);
    return flags;
}

int check_dims(int B, int K, int H, int D, int L, int Q, int P, int dtype) {
    if (dtype != MSDA_F32 && dtype != MSDA_F16 && dtype != MSDA_BF16) return MSDA_ERR_DTYPE;
    if (B <= 0 || K <= 0 || H <= 0 || D <= 0 || L <= 0 || Q <= 0 || P <= 0) return MSDA_ERR_DIMS;
    if (D > 256 || static_cast<long long>(L) * P > 64 || L > msda::kMaxLevels) return MSDA_ERR_LIMIT;
    const long long rows = static_cast<long long>(B) * K * H;
    const long long tasks = static_cast<long long>(B) * Q * H;
    if (rows >= (1LL << 31) || tasks >= (1LL << 31)) return MSDA_ERR_LIMIT;
    return MSDA_OK;
}

RowPlan plan_rows(int D, int dtype, bool ptrs_16B_aligned) {
    RowPlan rp{true, 32, 8};
    const size_t row_bytes = static_cast<size_t>(D) * elem_size(dtype);
    if (!ptrs_16B_aligned || row_bytes % 16 != 0) return rp;
    const int pieces = static_cast<int>(row_bytes / 16);
    if (pieces > 64) return rp;
    rp.scalar = false;
    rp.lpr = 1;
    while (rp.lpr < pieces && rp.lpr < 32) rp.lpr *= 2;
    rp.nv = (pieces + rp.lpr - 1) / rp.lpr;
    return rp;
}

// One past the last valid row offset.
uint32_t debug_limit(unsigned long long rows, unsigned long long units) {
#ifdef MSDA_DEBUG_BOUNDS
    // test hook of the bounds-checking build: pretend value / grad_value end after this many rows
    const unsigned long long pretend = static_cast<unsigned long long>(g_tune_debug_rows.load());
    if (pretend > 0 && pretend < rows) return static_cast<uint32_t>(pretend * units);
#endif
    return static_cast<uint32_t>(rows * units);
}

// Offsets of value rows travel as 32-bit counts of `row_units`: 16-byte pieces on the vector
// path, elements on the scalar path.
int set_row_units(Params& p, const RowPlan& rp, int dtype) {
    const unsigned long long units =
        rp.scalar ? static_cast<unsigned long long>(p.D)
                  : static_cast<unsigned long long>(p.D) * elem_size(dtype) / 16;
    const unsigned long long rows = static_cast<unsigned long long>(p.B) * p.K * p.H;
    if (rows * units >= 0xffffffffull) return MSDA_ERR_LIMIT;
    p.row_units = static_cast<uint32_t>(units);
    p.limit_units = debug_limit(rows, units);
    p.pieces = static_cast<int>(units);
    return MSDA_OK;
}

// Layout of the sorted backward's workspace: fp32 accumulation rows (16-bit tensors only),
// ticket counter, regions, sorted sample numbers; for the fused operator locations, weights and, 16-bit
// tensors only, their gradients.
struct SortPlan {
    size_t ticket, regions, sorted, loc, prob, grad_loc, grad_attn, total;
    uint32_t nsamples;
};

// False where the sorted backward does not apply: rows that are not whole groups of four
// channels, more samples than 32-bit counters hold.
bool plan_sort(int B, int K, int H, int D, int L, int Q, int P, int dtype, int mode, SortPlan* s) {
    if (D % 4 != 0) return false;
    const unsigned long long n = 1ull * B * Q * H * L * P;
    // ... nor as many tickets (regions of a few samples each get one)
    if (n + 1ull * B * H * L >= (1ull << 31) ||
        1ull * B * Q * H * (D / 4) >= (1ull << 32))
        return false;
    auto up = [](size_t v) { return (v + 255) / 256 * 256; };
    s->nsamples = static_cast<uint32_t>(n);
    s->ticket = dtype == MSDA_F32 ? 0 : up(static_cast<size_t>(B) * K * H * D * 4);
    s->regions = s->ticket + 256;
    s->sorted = s->regions + up(static_cast<size_t>(B) * H * L * sizeof(uint2));
    s->loc = s->sorted + up(n * 4);
    s->prob = s->loc + (mode == kFused ? up(n * 8) : 0);
    s->grad_loc = s->prob + (mode == kFused ? up(n * 4) : 0);
    const bool own = mode == kFused && dtype != MSDA_F32;
    s->grad_attn = s->grad_loc + (own ? up(n * 8) : 0);
    s->total = s->grad_attn + (own ? up(n * 4) : 0);
    return true;
}

// Where sorting pays: the gain is the rows that samples of one cell share, the cost a sort of 9 to 25 ps
// per sample, so it takes enough samples per cell, fewer of them the wider the rows, and enough samples for
// the tails of two more launches (four for the fused operator). A line per width: `least` million samples,
// `sparse` per cell and per_cell * millions^(3/4 or 3/2) >= `line`. The lines were drawn through 8000 calls
// of 0.1 to 30 M samples, 1.5 to 3000 per cell, one to five levels, 1 to 64 heads times images, locations
// uniform, around a grid or mostly outside: 1 to 4 % slower than the better form of each call (8 and 9 %
// for up to 16 channels of fp32 and for few samples of the fused operator). Whole backward on both sides of
// a line, millions of samples, per cell: unsorted / sorted (us); at 8 channels both occur beyond it, too
// (fp32 9.43, 16 per cell: 439/548; 16 bits 0.92, 24: 48/83):
//   width    fp32                                             16 bits
//   <= 8     0.49  61: 26/38    3.88  2.4: 243/291            1.76  10: 91/181   7.14   11: 365/464
//            0.40 168: 71/42    2.33   26: 294/163            0.81  26: 101/65   2.98   22: 183/138
//   <= 16    0.48  34: 40/42    1.88  5.2: 132/135            0.62  17: 50/58    1.19  4.1: 105/99
//            0.68  46: 99/56    2.42   10: 161/140            1.49  10: 118/97   2.50  6.0: 222/183
//   <= 32    0.35  53: 38/42    3.25  2.5: 361/388            0.33  28: 50/48    1.45  5.4: 150/134
//            0.60  35: 93/85    1.54  6.6: 323/214            0.53  58: 89/54    2.90  5.7: 306/275
//   <= 64    0.11 5.3: 38/46    0.72  1.5: 216/218            0.17  11: 48/48    0.85  2.7: 177/169
//            0.33 4.1: 79/60    1.66  1.9: 431/402            0.29  12: 73/56    2.49  2.9: 423/384
//   <= 128   0.30 2.0: 116/116  2.47  2.9: 937/730            0.10 4.2: 54/54    0.73  1.7: 257/261
//            0.26 2.0: 132/124  0.67  3.0: 274/230            0.18 3.5: 132/83   1.22  3.3: 519/374
//   <= 256   0.24 2.1: 226/159  1.65  4.2: 1281/572           0.14 1.6: 140/132  0.66  2.4: 701/394
//   fused    0.47  70: 60/68    2.13  2.0: 301/410  (<= 32)   0.56  75: 62/76    3.52  5.3: 405/388
//            0.87  32: 157/128  3.70   19: 720/458            1.74  27: 228/187  3.96   13: 511/394
//            0.11  34: 40/48    0.66  3.1: 151/153  (<= 64)   0.33  57: 62/70    2.68  2.6: 536/562
//            0.35  15: 89/76    1.23  2.5: 374/347            0.70  18: 126/102  2.80  3.1: 593/505
//            0.11  38: 60/75    0.21  2.1: 116/126  (<= 128)  0.33  2.7: 118/134 0.41  3.6: 140/142
//            0.20 7.0: 91/73    0.80  1.7: 378/332            0.23   23: 77/68   1.25  6.6: 343/276
// Up to 16 channels the two more kernels of the fused operator cost what the sort gains (1.28 M, 3.3 per
// cell 265/179, but 1.36 M, 4.7: 122/171). 16-bit rows that are not whole 16-byte pieces go through the
// unsorted kernel one channel at a time: sorted 2 to 16 times as fast from 1.5 per cell on. The
// nearest-pixel operator has one row per sample and no double-precision dot products: 519 / 397 at
// 24 x 107 k samples on 375 pixels.
struct SortLine {
    double least, sparse, line;
};
bool sort_pays(const SortPlan& s, int K, int H, int D, int dtype, int B, int mode) {
    if (g_tune_sort.load() == 0) return false;
    if (g_tune_sort.load() == 2) return true;
    if (s.nsamples < 100000u) return false;
    const double per_cell = static_cast<double>(s.nsamples) / (static_cast<double>(B) * K * H);
    if (mode == kNearest) return per_cell >= 16.0;
    const bool f32 = dtype == MSDA_F32;
    if (!f32 && D % 8 != 0) return per_cell >= 1.5;
    static const SortLine plain[2][6] = {
        {{0.1, 12.0, 15.0}, {0.1, 6.0, 15.0}, {0.5, 2.5, 10.0}, {0.1, 2.5, 2.5}, {0.1, 2.0, 0.6}, {0.1, 1.5, 0.5}},
        {{0.1, 12.0, 40.0}, {0.1, 6.0, 25.0}, {0.5, 6.0, 12.0}, {0.1, 1.5, 1.5}, {0.1, 1.5, 0.0}, {0.1, 1.5, 0.0}}};
    static const SortLine fused[2][4] = {
        {{0.8, 9.0, 30.0}, {0.5, 2.5, 9.0}, {0.2, 2.0, 1.3}, {0.1, 1.5, 0.15}},
        {{0.8, 9.0, 25.0}, {0.3, 1.5, 2.0}, {0.2, 1.5, 0.5}, {0.1, 1.5, 0.0}}};
    const int width = D <= 8 ? 0 : D <= 16 ? 1 : D <= 32 ? 2 : D <= 64 ? 3 : D <= 128 ? 4 : 5;
    if (mode == kFused && width < 2) return false;
    const SortLine& at = mode == kFused ? fused[f32][width - 2] : plain[f32][width];
    const double millions = 1e-6 * s.nsamples;
    return millions >= at.least && per_cell >= at.sparse &&
           per_cell * std::pow(millions, mode == kFused || width < 3 ? 1.5 : 0.75) >= at.line;
}

// Tasks that one warp pass takes together: as many as fill its lanes with samples, but fewer where
// there are so few tasks that `warps` take all of them in one round with fewer each (300 queries
// x 8 heads x 16 samples: forward 5.6 -> 4.5 us; with more rounds the fuller passes are faster).
int tasks_per_item(int LP, long long tasks, int warps) {
    if (LP >= msda::kChunk) return 1;
    const int most = msda::kChunk / LP;
    int t = 1;
    while (t < most && (tasks + t - 1) / t > warps) t *= 2;
    return t < most ? t : most;
}

// Fills the parts of Params common to both directions.
int fill_common(Params& p, const DeviceInfo* dev, const void* value, const int32_t* shapes,
                const int32_t* starts, const void* loc, const void* attn, int B, int K, int H,
                int D, int L, int Q, int P, int dtype, int table_flags, bool backward) {
    std::memset(&p, 0, sizeof(p));
    p.value = value;
    p.loc = loc;
    p.attn = attn;
    p.B = B; p.K = K; p.H = H; p.D = D; p.L = L; p.Q = Q; p.P = P;
    p.LP = L * P;
    p.tasks_per_item = tasks_per_item(p.LP, static_cast<long long>(B) * Q * H, dev->sm_count * (backward ? 24 : 32));
    p.ntasks = static_cast<long long>(B) * Q * H;
    p.nitems = (p.ntasks + p.tasks_per_item - 1) / p.tasks_per_item;
    p.status = dev->status_ptr;

    bool shapes_dev = true, starts_dev = true;
    if (!(table_flags & MSDA_TABLES_DEVICE)) {
        pointer_on_device(shapes, &shapes_dev);
        pointer_on_device(starts, &starts_dev);
    }
    const int step = (table_flags & MSDA_TABLES_INT64) ? 2 : 1;
    p.table_step = step;
    if (shapes_dev != starts_dev) return MSDA_ERR_ALIGN;  // both host or both device
    if (shapes_dev) {
        p.use_table = 0;
        p.shapes_dev = shapes;
        p.start_dev = starts;
    } else {
        p.use_table = 1;
        for (int l = 0; l < L; ++l) {
            p.lv.h[l] = shapes[2 * l * step];
            p.lv.w[l] = shapes[(2 * l + 1) * step];
            p.lv.start[l] = starts[l * step];
            if (p.lv.h[l] <= 0 || p.lv.w[l] <= 0 || p.lv.start[l] < 0 ||
                static_cast<long long>(p.lv.start[l]) + static_cast<long long>(p.lv.h[l]) * p.lv.w[l] > K)
                return MSDA_ERR_DIMS;
        }
    }
    const size_t e = elem_size(dtype);
    // Interleave the batch entries in the walk when all of value stays in L2 whatever the
    // order (16 MiB: measured neutral to harmful from 17 MiB up, a large gain for small maps), every entry holds a whole number of items, and the
    // counters fit the 32-bit fast division.
    p.walk_b = 0;
    p.walk_items_per_b = 0;
    p.fd_walk_b = msda::make_fastdiv(1);
    {
        const long long tasks_per_b = static_cast<long long>(Q) * H;
        const size_t value_bytes = static_cast<size_t>(B) * K * H * D * e;
        if (g_tune_interleave.load() != 0 && B > 1 && value_bytes <= (16u << 20) &&
            tasks_per_b % p.tasks_per_item == 0 && p.nitems < (1ll << 31)) {
            p.walk_b = static_cast<uint32_t>(B);
            p.walk_items_per_b = static_cast<uint32_t>(tasks_per_b / p.tasks_per_item);
            p.fd_walk_b = msda::make_fastdiv(static_cast<uint32_t>(B));
        }
    }
    p.fd_qh = msda::make_fastdiv(static_cast<uint32_t>(Q) * static_cast<uint32_t>(H));
    p.fd_h = msda::make_fastdiv(static_cast<uint32_t>(H));
    p.fd_lp = msda::make_fastdiv(static_cast<uint32_t>(p.LP));
    // Bulk-copy staging needs 16-byte aligned sources and sizes: per item the weights take
    // samples * e bytes and the locations twice that.
    const size_t item_attn_bytes = static_cast<size_t>(p.tasks_per_item) * p.LP * e;
    const int stage_mode = g_tune_stage.load();
    p.stage = ((stage_mode == 1 || (stage_mode == 2 && backward)) && aligned_to(loc, 16) &&
               aligned_to(attn, 16) && item_attn_bytes % 16 == 0)
                  ? 1
                  : 0;
    p.spin_limit = g_tune_spin.load();
    p.pack_rows = g_tune_pack.load() != 0 ? 1 : 0;
    p.precise_amp = static_cast<float>(g_tune_precise_amp.load());
    if (!aligned_to(value, e) || !aligned_to(loc, e) || !aligned_to(attn, e)) return MSDA_ERR_ALIGN;
    return MSDA_OK;
}

int backward_impl(const void* value, const int32_t* shapes, const int32_t* starts, const void* loc,
                  const void* attn, const void* grad_out, void* grad_value, void* grad_loc,
                  void* grad_attn, void* workspace, size_t workspace_bytes, bool use_ws, int mode,
                  const void* ref, float* grad_ref, int B, int K, int H, int D, int L, int Q,
                  int P, int dtype, void* stream_v) {
    // mode: kBilinear = MSDA; kNearest = geometric kernel attention (one clamped integer pixel
    // per sample, no location gradient); kFused = MSDA fed by reference points, offsets (in
    // `loc`) and logits (in `attn`)
    const bool nearest = mode == kNearest;
    const int table_flags = split_flags(&dtype);
    if (!value || !shapes || !starts || !loc || !attn || !grad_out || !grad_value || !grad_attn ||
        (!nearest && !grad_loc) || (mode == kFused && (!ref || !grad_ref)))
        return MSDA_ERR_NULL;
    if (mode == kFused && static_cast<long long>(L) * P > 32) return MSDA_ERR_LIMIT;
    int rc = check_dims(B, K, H, D, L, Q, P, dtype);
    if (rc != MSDA_OK) return rc;
    const DeviceInfo* dev = nullptr;
    rc = device_info(&dev);
    if (rc != MSDA_OK) return rc;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);

    Params p;
    rc = fill_common(p, dev, value, shapes, starts, loc, attn, B, K, H, D, L, Q, P, dtype,
                     table_flags, true);
    if (rc != MSDA_OK) return rc;
    const size_t e = elem_size(dtype);
    if (!aligned_to(grad_out, e) || !aligned_to(grad_value, e) || !aligned_to(grad_attn, e) ||
        (!nearest && !aligned_to(grad_loc, 2 * e)))
        return MSDA_ERR_ALIGN;

    const long long nval = static_cast<long long>(B) * K * H * D;
    const bool acc_f32 = use_ws && dtype != MSDA_F32;
    // the sorted form, where the caller brought the workspace for it
    SortPlan plan;
    if (use_ws && plan_sort(B, K, H, D, L, Q, P, dtype, mode, &plan) &&
        sort_pays(plan, K, H, D, dtype, B, mode) &&
        workspace && workspace_bytes >= plan.total && aligned_to(workspace, 16) &&
        aligned_to(value, 4 * e) && aligned_to(grad_out, 4 * e) &&
        aligned_to(acc_f32 ? workspace : grad_value, 16) && aligned_to(loc, 2 * e)) {
        char* ws = static_cast<char*>(workspace);
        float* acc = static_cast<float*>(acc_f32 ? workspace : grad_value);
        const unsigned long long quads = static_cast<unsigned long long>(D) / 4;
        if (static_cast<unsigned long long>(B) * K * H * quads < 0xffffffffull) {
            p.row_units = static_cast<uint32_t>(quads);
            p.limit_units = debug_limit(static_cast<unsigned long long>(B) * K * H, quads);
            p.grad_out = grad_out;
            p.grad_value = acc;
            p.grad_loc = grad_loc;
            p.grad_attn = grad_attn;
            msda::SortParams sp{};
            sp.ticket = reinterpret_cast<uint32_t*>(ws + plan.ticket);
            sp.regions = reinterpret_cast<uint2*>(ws + plan.regions);
            sp.sorted = reinterpret_cast<uint32_t*>(ws + plan.sorted);
            sp.nsamples = plan.nsamples;
            sp.fd_p = msda::make_fastdiv(static_cast<uint32_t>(P));
            const msda::LaunchShape shape{dev->sm_count, g_tune_cps_bwd.load()};
            cudaError_t ce = cudaSuccess;   // (the launch of the sort sees to the zeros in acc)
            prof_record(2, stream);
            if (mode == kFused) {
                p.ref = ref;
                p.grad_ref = grad_ref;
                msda::FusedSamples fs;
                fs.loc = reinterpret_cast<float2*>(ws + plan.loc);
                fs.prob = reinterpret_cast<float*>(ws + plan.prob);
                fs.grad_loc = acc_f32 ? reinterpret_cast<float2*>(ws + plan.grad_loc) : static_cast<float2*>(grad_loc);
                fs.grad_attn = acc_f32 ? reinterpret_cast<float*>(ws + plan.grad_attn) : static_cast<float*>(grad_attn);
                ce = cudaMemsetAsync(grad_ref, 0, static_cast<size_t>(B) * Q * L * 2 * sizeof(float), stream);
                if (ce == cudaSuccess)
                    ce = msda::launch_fused_backward_sorted(p, sp, fs, dtype, shape, stream);
            } else {
                ce = nearest ? msda::launch_gka_backward_sorted(p, sp, dtype, shape, stream)
                             : msda::launch_backward_sorted(p, sp, dtype, shape, stream);
            }
            prof_record(3, stream);
            if (ce != cudaSuccess) return fail_cuda(ce);
            g_launches.fetch_add(mode == kFused ? 4 : 2, std::memory_order_relaxed);
            if (acc_f32) {
                ce = msda::launch_downcast(acc, grad_value, nval, dtype, stream);
                if (ce != cudaSuccess) return fail_cuda(ce);
                g_launches.fetch_add(1, std::memory_order_relaxed);
            }
            return MSDA_OK;
        }
    }
    void* acc = grad_value;
    size_t acc_bytes = static_cast<size_t>(nval) * e;
    if (acc_f32) {
        const size_t need = static_cast<size_t>(nval) * sizeof(float);
        if (!workspace || workspace_bytes < need || !aligned_to(workspace, 16))
            return MSDA_ERR_WORKSPACE;
        acc = workspace;
        acc_bytes = need;
    }
    const bool vec_ok = aligned_to(value, 16) && aligned_to(grad_out, 16) && aligned_to(acc, 16);
    const RowPlan rp = plan_rows(D, dtype, vec_ok);

    rc = set_row_units(p, rp, dtype);
    if (rc != MSDA_OK) return rc;
    p.warp_smem = msda::bwd_warp_smem(p.tasks_per_item * p.LP, e);
    p.grad_out = grad_out;
    p.grad_value = acc;
    p.grad_loc = grad_loc;
    p.grad_attn = grad_attn;

    cudaError_t ce = cudaMemsetAsync(acc, 0, acc_bytes, stream);
    if (ce != cudaSuccess) return fail_cuda(ce);
    prof_record(2, stream);
    const msda::LaunchShape shape{dev->sm_count, g_tune_cps_bwd.load()};
    if (mode == kFused) {
        p.ref = ref;
        p.grad_ref = grad_ref;
        ce = cudaMemsetAsync(grad_ref, 0, static_cast<size_t>(B) * Q * L * 2 * sizeof(float),
                             stream);
        if (ce != cudaSuccess) return fail_cuda(ce);
        ce = msda::launch_fused_backward(p, dtype, acc_f32 ? 1 : 0, rp, shape, stream);
    } else if (nearest) {
        ce = msda::launch_gka_backward(p, dtype, acc_f32 ? 1 : 0, rp, shape, stream);
    } else {
        ce = msda::launch_backward(p, dtype, acc_f32 ? 1 : 0, rp, shape, stream);
    }
    prof_record(3, stream);
    if (ce != cudaSuccess) return fail_cuda(ce);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    if (acc_f32) {
        ce = msda::launch_downcast(static_cast<const float*>(acc), grad_value, nval, dtype, stream);
        if (ce != cudaSuccess) return fail_cuda(ce);
        g_launches.fetch_add(1, std::memory_order_relaxed);
    }
    return MSDA_OK;
}

int forward_impl(const void* value, const int32_t* spatial_shapes,
                 const int32_t* level_start_index, const void* sampling_locations,
                 const void* attention_weights, void* output, int mode, const void* ref, int B,
                 int K, int H, int D, int L, int Q, int P, int dtype, void* stream_v) {
    const int table_flags = split_flags(&dtype);
    if (mode == kFused && (!ref || static_cast<long long>(L) * P > 32))
        return ref ? MSDA_ERR_LIMIT : MSDA_ERR_NULL;
    if (!value || !spatial_shapes || !level_start_index || !sampling_locations ||
        !attention_weights || !output)
        return MSDA_ERR_NULL;
    int rc = check_dims(B, K, H, D, L, Q, P, dtype);
    if (rc != MSDA_OK) return rc;
    const DeviceInfo* dev = nullptr;
    rc = device_info(&dev);
    if (rc != MSDA_OK) return rc;

    Params p;
    rc = fill_common(p, dev, value, spatial_shapes, level_start_index, sampling_locations,
                     attention_weights, B, K, H, D, L, Q, P, dtype, table_flags, false);
    if (rc != MSDA_OK) return rc;
    if (!aligned_to(output, elem_size(dtype))) return MSDA_ERR_ALIGN;
    p.out = output;
    const RowPlan rp = plan_rows(D, dtype, aligned_to(value, 16) && aligned_to(output, 16));
    rc = set_row_units(p, rp, dtype);
    if (rc != MSDA_OK) return rc;
    p.warp_smem = msda::fwd_warp_smem(p.tasks_per_item * p.LP, elem_size(dtype));
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    prof_record(0, stream);
    const msda::LaunchShape shape{dev->sm_count, g_tune_cps_fwd.load()};
    p.ref = ref;
    cudaError_t ce = mode == kFused     ? msda::launch_fused_forward(p, dtype, rp, shape, stream)
                     : mode == kNearest ? msda::launch_gka_forward(p, dtype, rp, shape, stream)
                                        : msda::launch_forward(p, dtype, rp, shape, stream);
    prof_record(1, stream);
    if (ce != cudaSuccess) return fail_cuda(ce);
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return MSDA_OK;
}

}  // namespace

namespace msda {
void count_launches(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
int note_cuda_error(cudaError_t e) { return fail_cuda(e); }
int device_facts(int* sm_count, int** status_word) {
    const DeviceInfo* d = nullptr;
    const int rc = device_info(&d);
    if (rc != MSDA_OK) return rc;
    if (sm_count != nullptr) *sm_count = d->sm_count;
    if (status_word != nullptr) *status_word = d->status_ptr;
    return MSDA_OK;
}
}  // namespace msda

extern "C" {

int msda_sm100_forward(const void* value, const int32_t* spatial_shapes,
                       const int32_t* level_start_index, const void* sampling_locations,
                       const void* attention_weights, void* output, int B, int K, int H, int D,
                       int L, int Q, int P, int dtype, void* stream) {
    return forward_impl(value, spatial_shapes, level_start_index, sampling_locations,
                        attention_weights, output, kBilinear, nullptr, B, K, H, D, L, Q, P, dtype,
                        stream);
}

int gka_sm100_forward(const void* value, const int32_t* spatial_shapes,
                      const int32_t* level_start_index, const void* sampling_locations,
                      const void* attention_weights, void* output, int B, int K, int H, int D,
                      int L, int Q, int P, int dtype, void* stream) {
    return forward_impl(value, spatial_shapes, level_start_index, sampling_locations,
                        attention_weights, output, kNearest, nullptr, B, K, H, D, L, Q, P, dtype,
                        stream);
}

int msda_sm100_fused_forward(const void* value, const int32_t* spatial_shapes,
                             const int32_t* level_start_index, const void* reference_points,
                             const void* sampling_offsets, const void* attention_logits,
                             void* output, int B, int K, int H, int D, int L, int Q, int P,
                             int dtype, void* stream) {
    return forward_impl(value, spatial_shapes, level_start_index, sampling_offsets,
                        attention_logits, output, kFused, reference_points, B, K, H, D, L, Q, P,
                        dtype, stream);
}

int msda_sm100_fused_backward_ws(const void* value, const int32_t* spatial_shapes,
                                 const int32_t* level_start_index, const void* reference_points,
                                 const void* sampling_offsets, const void* attention_logits,
                                 const void* grad_output, void* grad_value,
                                 float* grad_reference_points, void* grad_sampling_offsets,
                                 void* grad_attention_logits, void* workspace,
                                 size_t workspace_bytes, int B, int K, int H, int D, int L, int Q,
                                 int P, int dtype, void* stream) {
    return backward_impl(value, spatial_shapes, level_start_index, sampling_offsets,
                         attention_logits, grad_output, grad_value, grad_sampling_offsets,
                         grad_attention_logits, workspace, workspace_bytes, true, kFused,
                         reference_points, grad_reference_points, B, K, H, D, L, Q, P, dtype,
                         stream);
}

int gka_sm100_backward_ws(const void* value, const int32_t* spatial_shapes,
                          const int32_t* level_start_index, const void* sampling_locations,
                          const void* attention_weights, const void* grad_output,
                          void* grad_value, void* grad_attn_weight, void* workspace,
                          size_t workspace_bytes, int B, int K, int H, int D, int L, int Q, int P,
                          int dtype, void* stream) {
    return backward_impl(value, spatial_shapes, level_start_index, sampling_locations,
                         attention_weights, grad_output, grad_value, nullptr, grad_attn_weight,
                         workspace, workspace_bytes, true, kNearest, nullptr, nullptr, B, K, H, D,
                         L, Q, P, dtype, stream);
}

int msda_sm100_backward(const void* value, const int32_t* spatial_shapes,
                        const int32_t* level_start_index, const void* sampling_locations,
                        const void* attention_weights, const void* grad_output, void* grad_value,
                        void* grad_sampling_loc, void* grad_attn_weight, int B, int K, int H,
                        int D, int L, int Q, int P, int dtype, void* stream) {
    return backward_impl(value, spatial_shapes, level_start_index, sampling_locations,
                         attention_weights, grad_output, grad_value, grad_sampling_loc,
                         grad_attn_weight, nullptr, 0, false, kBilinear, nullptr, nullptr, B, K, H, D, L,
                         Q, P, dtype, stream);
}

size_t msda_sm100_backward_workspace_bytes(int B, int K, int H, int D, int dtype) {
    if (dtype == MSDA_F32 || B <= 0 || K <= 0 || H <= 0 || D <= 0) return 0;
    return static_cast<size_t>(B) * K * H * D * sizeof(float);
}

static size_t sorted_workspace(int B, int K, int H, int D, int L, int Q, int P, int dtype, int mode) {
    SortPlan plan;
    if (check_dims(B, K, H, D, L, Q, P, dtype) != MSDA_OK ||
        !plan_sort(B, K, H, D, L, Q, P, dtype, mode, &plan) || !sort_pays(plan, K, H, D, dtype, B, mode))
        return msda_sm100_backward_workspace_bytes(B, K, H, D, dtype);
    return plan.total;
}

size_t msda_sm100_backward_sorted_workspace_bytes(int B, int K, int H, int D, int L, int Q, int P,
                                                  int dtype) {
    return sorted_workspace(B, K, H, D, L, Q, P, dtype, kBilinear);
}

size_t msda_sm100_fused_backward_sorted_workspace_bytes(int B, int K, int H, int D, int L, int Q, int P,
                                                        int dtype) {
    return sorted_workspace(B, K, H, D, L, Q, P, dtype, kFused);
}

size_t gka_sm100_backward_sorted_workspace_bytes(int B, int K, int H, int D, int L, int Q, int P,
                                                 int dtype) {
    return sorted_workspace(B, K, H, D, L, Q, P, dtype, kNearest);
}

int msda_sm100_backward_ws(const void* value, const int32_t* spatial_shapes,
                           const int32_t* level_start_index, const void* sampling_locations,
                           const void* attention_weights, const void* grad_output,
                           void* grad_value, void* grad_sampling_loc, void* grad_attn_weight,
                           void* workspace, size_t workspace_bytes, int B, int K, int H, int D,
                           int L, int Q, int P, int dtype, void* stream) {
    return backward_impl(value, spatial_shapes, level_start_index, sampling_locations,
                         attention_weights, grad_output, grad_value, grad_sampling_loc,
                         grad_attn_weight, workspace, workspace_bytes, true, kBilinear, nullptr, nullptr,
                         B, K, H, D, L, Q, P, dtype, stream);
}

size_t msda_sm100_forward_bytes(int B, int K, int H, int D, int L, int Q, int P, int dtype) {
    const size_t e = elem_size(dtype);
    const size_t v = static_cast<size_t>(B) * K * H * D;
    const size_t s = static_cast<size_t>(B) * Q * H * L * P;
    const size_t o = static_cast<size_t>(B) * Q * H * D;
    return e * (v + 3 * s + o);
}

size_t msda_sm100_backward_bytes(int B, int K, int H, int D, int L, int Q, int P, int dtype) {
    const size_t e = elem_size(dtype);
    const size_t v = static_cast<size_t>(B) * K * H * D;
    const size_t s = static_cast<size_t>(B) * Q * H * L * P;
    const size_t o = static_cast<size_t>(B) * Q * H * D;
    return e * (2 * v + 6 * s + o);
}

int msda_sm100_device_status(int clear) {
    const DeviceInfo* dev = nullptr;
    int rc = device_info(&dev);
    if (rc != MSDA_OK) return rc;
    cudaError_t ce = cudaDeviceSynchronize();
    if (ce != cudaSuccess) return fail_cuda(ce);
    int word = 0;
    ce = cudaMemcpy(&word, dev->status_ptr, sizeof(int), cudaMemcpyDeviceToHost);
    if (ce != cudaSuccess) return fail_cuda(ce);
    if (clear) {
        ce = cudaMemset(dev->status_ptr, 0, sizeof(int));
        if (ce != cudaSuccess) return fail_cuda(ce);
    }
    return word;
}

int msda_sm100_sort_form(int maps, int samples, int mean_cells, int most_cells, int cells, int sm_count) {
    if (maps <= 0 || samples <= 0 || mean_cells < 0 || most_cells <= 0 || cells <= 0 || sm_count <= 0)
        return MSDA_ERR_DIMS;
    const uint32_t n = static_cast<uint32_t>(samples), c = static_cast<uint32_t>(cells);
    const msda::SortChoice s = msda::choose_sort(
        {static_cast<uint32_t>(maps), n, static_cast<uint32_t>(mean_cells), static_cast<uint32_t>(most_cells)},
        static_cast<uint32_t>(sm_count), false);
    const msda::Counters kept = msda::counters_of(s.parts, n, c);
    const bool staged = kept == msda::Counters::kAlone && c + (n - 1) / s.parts + 1 <= s.room;
    return static_cast<int>(s.parts) | static_cast<int>(kept) << 4 | (staged ? 64 : 0) |
           (s.room > msda::kSortCells ? 128 : 0);
}

int msda_sm100_tune(int knob, int value) {
    std::atomic<int>* target = nullptr;
    switch (knob) {
        case MSDA_TUNE_STAGE: target = &g_tune_stage; break;
        case MSDA_TUNE_CTAS_PER_SM: target = &g_tune_cps_fwd; break;
        case MSDA_TUNE_CTAS_PER_SM_BWD: target = &g_tune_cps_bwd; break;
        case MSDA_TUNE_INTERLEAVE: target = &g_tune_interleave; break;
        case MSDA_TUNE_SPIN_LIMIT: target = &g_tune_spin; break;
        case MSDA_TUNE_PRECISE_AMP: target = &g_tune_precise_amp; break;
        case MSDA_TUNE_DEBUG_ROW_LIMIT: target = &g_tune_debug_rows; break;
        case MSDA_TUNE_PACK_ROWS: target = &g_tune_pack; break;
        case MSDA_TUNE_SORT: target = &g_tune_sort; break;
        default: return MSDA_ERR_DIMS;
    }
    if (value < 0) return target->load();
    return target->exchange(value);
}

void msda_sm100_profile_events(void* fwd_start, void* fwd_stop, void* bwd_start, void* bwd_stop) {
    t_prof[0] = static_cast<cudaEvent_t>(fwd_start);
    t_prof[1] = static_cast<cudaEvent_t>(fwd_stop);
    t_prof[2] = static_cast<cudaEvent_t>(bwd_start);
    t_prof[3] = static_cast<cudaEvent_t>(bwd_stop);
}

long long msda_sm100_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }

const char* msda_sm100_strerror(int status) {
    switch (status) {
        case MSDA_OK: return "ok";
        case MSDA_ERR_NULL: return "a required pointer is NULL";
        case MSDA_ERR_DIMS: return "a dimension or level shape is out of range";
        case MSDA_ERR_LIMIT: return "limit exceeded (D <= 256, L*P <= 64, indices < 2^31)";
        case MSDA_ERR_ALIGN: return "a pointer is misaligned for its element type";
        case MSDA_ERR_DTYPE: return "unknown dtype code";
        case MSDA_ERR_WORKSPACE: return "workspace missing, misaligned or too small";
        case MSDA_ERR_CUDA: return "a CUDA runtime call failed";
        default: return "unknown status";
    }
}

int msda_sm100_last_cuda_error(void) { return t_last_cuda_error; }

int msda_sm100_abi_version(void) { return kAbiVersion; }

int msda_sm100_debug_bounds(void) {
#ifdef MSDA_DEBUG_BOUNDS
    return 1;
#else
    return 0;
#endif
}

}  // extern "C"
