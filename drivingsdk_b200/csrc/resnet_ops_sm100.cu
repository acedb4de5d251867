// Element-wise add + ReLU (with its gradient) and the 3x3 / stride-2 / pad-1 max pooling of a
// ResNet stem, for sm_100a. Both are pure streaming work: the only figure of merit is the share
// of HBM bandwidth they reach, so every thread moves 16 bytes per access and keeps four
// independent accesses in flight.
//
// Replaces aclnnAddRelu + ReluGrad (mx_driving/csrc/AddRelu.cpp:20-32) and
// aclnnMaxPool2dWithMask / aclnnMaxPool2d (mx_driving/csrc/MaxPool2d.cpp:45-100).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "../../include/conv_ops_sm100.h"
#include "msda_launch.h"

namespace {

constexpr int kThreads = 256;
constexpr int kVecPerThread = 4;  // 16-byte accesses in flight per thread and operand

template <typename T> struct Cvt;
template <> struct Cvt<float> {
    static __device__ __forceinline__ float up(float v) { return v; }
    static __device__ __forceinline__ float down(float v) { return v; }
};
template <> struct Cvt<__half> {
    static __device__ __forceinline__ float up(__half v) { return __half2float(v); }
    static __device__ __forceinline__ __half down(float v) { return __float2half_rn(v); }
};
template <> struct Cvt<__nv_bfloat16> {
    static __device__ __forceinline__ float up(__nv_bfloat16 v) { return __bfloat162float(v); }
    static __device__ __forceinline__ __nv_bfloat16 down(float v) { return __float2bfloat16_rn(v); }
};

// relu that keeps NaN: (v > 0) is false for NaN, so select on !(v <= 0)
__device__ __forceinline__ float relu_keep_nan(float v) { return (v <= 0.f) ? 0.f : v; }

template <typename T> struct alignas(16) Vec16 {
    static constexpr int kN = 16 / sizeof(T);
    T v[kN];
};

// BACKWARD == false: relu(a + b) written to `dst` (may be a)
// BACKWARD == true : dst = a > 0 ? b : 0          (a = forward result, b = grad_out)
template <typename T, bool BACKWARD>
__device__ __forceinline__ T combine(T a, T b) {
    if (BACKWARD) return (Cvt<T>::up(a) > 0.f) ? b : Cvt<T>::down(0.f);
    return Cvt<T>::down(relu_keep_nan(Cvt<T>::up(a) + Cvt<T>::up(b)));
}

template <typename T, bool BACKWARD>
__global__ void __launch_bounds__(kThreads)
pointwise_vec_kernel(const T* a, const T* __restrict__ b, T* dst,  // a may alias dst
                     size_t nvec) {
    using V = Vec16<T>;
    const V* av = reinterpret_cast<const V*>(a);
    const V* bv = reinterpret_cast<const V*>(b);
    V* dv = reinterpret_cast<V*>(dst);
    const size_t tile = static_cast<size_t>(kThreads) * kVecPerThread;
    for (size_t base = static_cast<size_t>(blockIdx.x) * tile; base < nvec;
         base += static_cast<size_t>(gridDim.x) * tile) {
        V ra[kVecPerThread], rb[kVecPerThread];
#pragma unroll
        for (int u = 0; u < kVecPerThread; ++u) {
            const size_t i = base + static_cast<size_t>(u) * kThreads + threadIdx.x;
            if (i < nvec) {
                ra[u] = av[i];
                rb[u] = bv[i];
            }
        }
#pragma unroll
        for (int u = 0; u < kVecPerThread; ++u) {
            const size_t i = base + static_cast<size_t>(u) * kThreads + threadIdx.x;
            if (i < nvec) {
                V r;
#pragma unroll
                for (int k = 0; k < V::kN; ++k) r.v[k] = combine<T, BACKWARD>(ra[u].v[k], rb[u].v[k]);
                dv[i] = r;
            }
        }
    }
}

// elements [first, n): the tail after the last whole 16 bytes, or everything when a pointer
// is not 16-byte aligned
template <typename T, bool BACKWARD>
__global__ void __launch_bounds__(kThreads)
pointwise_scalar_kernel(const T* a, const T* __restrict__ b, T* dst,
                        size_t first, size_t n) {
    for (size_t i = first + static_cast<size_t>(blockIdx.x) * kThreads + threadIdx.x; i < n;
         i += static_cast<size_t>(gridDim.x) * kThreads)
        dst[i] = combine<T, BACKWARD>(a[i], b[i]);
}

template <typename T, bool BACKWARD>
int launch_pointwise(const void* a, const void* b, void* dst, size_t n, cudaStream_t stream) {
    int sms = 0;
    const int rc = msda::device_facts(&sms, nullptr);
    if (rc != MSDA_OK) return rc;
    const T* ap = static_cast<const T*>(a);
    const T* bp = static_cast<const T*>(b);
    T* dp = static_cast<T*>(dst);
    const bool aligned = ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) |
                           reinterpret_cast<uintptr_t>(dst)) % 16) == 0;
    const size_t per_vec = 16 / sizeof(T);
    const size_t nvec = aligned ? n / per_vec : 0;
    int launches = 0;
    if (nvec > 0) {
        const size_t tile = static_cast<size_t>(kThreads) * kVecPerThread;
        const size_t want = (nvec + tile - 1) / tile;
        const size_t cap = static_cast<size_t>(sms) * 8;  // 8 resident CTAs of 256 threads per SM
        const unsigned grid = static_cast<unsigned>(want < cap ? want : cap);
        pointwise_vec_kernel<T, BACKWARD><<<grid, kThreads, 0, stream>>>(ap, bp, dp, nvec);
        ++launches;
    }
    const size_t first = nvec * per_vec;
    if (first < n) {
        const size_t want = (n - first + kThreads - 1) / kThreads;
        const size_t cap = static_cast<size_t>(sms) * 8;
        const unsigned grid = static_cast<unsigned>(want < cap ? want : cap);
        pointwise_scalar_kernel<T, BACKWARD><<<grid, kThreads, 0, stream>>>(ap, bp, dp, first, n);
        ++launches;
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return msda::note_cuda_error(e);
    msda::count_launches(launches);
    return MSDA_OK;
}

template <bool BACKWARD>
int dispatch_pointwise(const void* a, const void* b, void* dst, size_t n, int dtype,
                       void* stream) {
    if (a == nullptr || b == nullptr || dst == nullptr) return MSDA_ERR_NULL;
    if (n == 0) return MSDA_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    switch (dtype) {
        case MSDA_F32: return launch_pointwise<float, BACKWARD>(a, b, dst, n, s);
        case MSDA_F16: return launch_pointwise<__half, BACKWARD>(a, b, dst, n, s);
        case MSDA_BF16: return launch_pointwise<__nv_bfloat16, BACKWARD>(a, b, dst, n, s);
        default: return MSDA_ERR_DTYPE;
    }
}

// ---------------------------------------------------------------------------------------------
// 3x3 / stride 2 / pad 1 max pooling, NCHW; bound by reading x once. A thread produces COLS
// neighbouring outputs of R output rows, which share all but the outermost of their 2 R + 1 input rows,
// and asks for all of its inputs before it uses the first. The column to the left comes from the
// neighbouring lane. COLS = 4 reads 16 bytes at a time and needs rows that start on 16 bytes
// (6 x 64 x 464 x 800: fp32 111 us, 0.98 of the copy rate, fp16 64; one output row per thread with 64-bit
// divisions and looser loads took 133 and 120); other widths and addresses take COLS = 1, whose loads of
// every other element meet the same cache lines (6 x 64 x 464 x 799 fp32 235 -> 126 us, fp16 148 -> 112).
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ float max_nan(float a, float b) {   // NaN if either is
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}

struct PoolGrid {
    int H, W, OH, OW;
    uint32_t groups, strips, total;            // of COLS outputs in a row; of R output rows; threads
    int first_row;                             // output row of the first thread
    msda::FastDiv by_groups, by_strips;
};

template <typename T, int COLS, int R>
__global__ void __launch_bounds__(kThreads)
maxpool3s2_kernel(const T* __restrict__ x, T* __restrict__ y, const __grid_constant__ PoolGrid p,
                  int vec_out) {
    constexpr int kPerVec = 16 / sizeof(T);                  // elements per 16-byte load
    constexpr int kPieces = COLS == 4 ? 8 / kPerVec : 1;     // loads of a thread in a row
    constexpr int kRows = 2 * R + 1;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t n = blockIdx.x * kThreads + threadIdx.x;
    const uint32_t idx = min(n, p.total - 1u);               // (all lanes take part in the shuffles)
    const uint32_t t = msda::fd_div(idx, p.by_groups), gq = idx - t * p.groups;
    const uint32_t plane = msda::fd_div(t, p.by_strips);     // n * C + c
    const int oh0 = p.first_row + static_cast<int>(t - plane * p.strips) * R;
    const int ow0 = static_cast<int>(gq) * COLS, c0 = 2 * ow0;
    const T* src = x + plane * (static_cast<size_t>(p.H) * p.W) + c0;

    const T lowest = Cvt<T>::down(-INFINITY);
    alignas(16) T raw[kRows][COLS == 4 ? 8 : 2];
    T before[kRows];
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
        const int h = 2 * oh0 - 1 + i;
        const bool in = h >= 0 && h < p.H;
        const T* row = src + static_cast<ptrdiff_t>(h) * p.W;
        if constexpr (COLS == 4) {
#pragma unroll
            for (int q = 0; q < kPieces; ++q) {
                if (in && c0 + q * kPerVec < p.W) {          // (a whole piece then)
                    *reinterpret_cast<uint4*>(&raw[i][q * kPerVec]) =
                        __ldg(reinterpret_cast<const uint4*>(row + q * kPerVec));
                } else {
#pragma unroll
                    for (int j = 0; j < kPerVec; ++j) raw[i][q * kPerVec + j] = lowest;
                }
            }
        } else {
            raw[i][0] = in ? row[0] : lowest;
            raw[i][1] = in && c0 + 1 < p.W ? row[1] : lowest;
        }
        before[i] = in && lane == 0 && gq > 0 ? row[-1] : lowest;
    }
    float m[kRows][COLS];   // of a row's three columns
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
        float left = __shfl_up_sync(0xffffffffu, Cvt<T>::up(raw[i][2 * COLS - 1]), 1);
        if (lane == 0 || gq == 0) left = Cvt<T>::up(before[i]);
#pragma unroll
        for (int o = 0; o < COLS; ++o) {
            const float a = Cvt<T>::up(raw[i][2 * o]), b = Cvt<T>::up(raw[i][2 * o + 1]);
            m[i][o] = max_nan(max_nan(left, a), b);
            left = b;
        }
    }
    if (n >= p.total) return;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int oh = oh0 + r;
        if (oh >= p.OH) break;
        T* dst = y + (plane * static_cast<size_t>(p.OH) + oh) * p.OW + ow0;
        alignas(16) T out[COLS];
#pragma unroll
        for (int o = 0; o < COLS; ++o) {
            const float v = max_nan(max_nan(m[2 * r][o], m[2 * r + 1][o]), m[2 * r + 2][o]);
            out[o] = Cvt<T>::down(v != v ? __int_as_float(0x7fc00000) : v);
        }
        if (COLS == 4 && vec_out && ow0 + 3 < p.OW) {
            if (sizeof(T) == 4) *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<uint4*>(out);
            else *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<uint2*>(out);
        } else {
#pragma unroll
            for (int o = 0; o < COLS; ++o)
                if (ow0 + o < p.OW) dst[o] = out[o];
        }
    }
}

template <typename T>
int launch_maxpool(const T* x, T* y, size_t planes, int H, int W, cudaStream_t stream) {
    // 16-byte loads need every row to start on a 16-byte boundary; vector stores likewise
    const int per_vec = 16 / static_cast<int>(sizeof(T));
    const bool vec_in = (reinterpret_cast<uintptr_t>(x) % 16 == 0) && (W % per_vec == 0);
    PoolGrid p;
    p.H = H; p.W = W; p.OH = (H - 1) / 2 + 1; p.OW = (W - 1) / 2 + 1;
    p.groups = static_cast<uint32_t>((p.OW - 1) / (vec_in ? 4 : 1) + 1);
    p.by_groups = msda::make_fastdiv(p.groups);
    // Rows of a thread: two of fp32, or four single outputs, unless the plane has few rows or the threads
    // would be few (32 x 104 x 104 fp32 3.7 us with two, 3.2 with one; 64000 x 8 x 8 9.3 and 7.2; 400 K x
    // 3 x 3 9.6 with four, 7.5 with two). In 16 bits one row is never slower than two or four (6 x 64 x 464 x
    // 800 67 us with four, 63 with one; 512 x 56 x 56 4.0 and 3.1).
    int rows = !vec_in ? 4 : sizeof(T) == 4 ? 2 : 1;
    auto strips = [&](int r) { return static_cast<uint32_t>((p.OH - 1) / r + 1); };
    while (rows > 1 && ((vec_in ? 2 * rows : rows / 2) >= p.OH || planes * strips(rows) * p.groups < (1u << 16)))
        rows /= 2;
    p.strips = strips(rows);
    p.by_strips = msda::make_fastdiv(p.strips);
    const int vec_out = (reinterpret_cast<uintptr_t>(y) % 16 == 0) && (p.OW % 4 == 0);
    auto kernel = vec_in ? (rows == 1 ? maxpool3s2_kernel<T, 4, 1> : maxpool3s2_kernel<T, 4, sizeof(T) == 4 ? 2 : 1>)
                         : (rows == 1   ? maxpool3s2_kernel<T, 1, 1>
                            : rows == 2 ? maxpool3s2_kernel<T, 1, 2>
                                        : maxpool3s2_kernel<T, 1, 4>);
    // FastDiv takes 2^31 - 1 threads: nearly always one launch, else some planes at a time, or some strips
    // of one where a plane has more
    const size_t most = (1u << 31) - 1, all = planes * p.strips, whole = most / p.groups / p.strips;
    int launches = 0;
    for (size_t first = 0; first < all; ++launches) {
        const size_t plane = first / p.strips, strip = first - plane * p.strips;
        const size_t count = whole > 0 ? std::min(whole, planes - plane) * p.strips
                                       : std::min(most / p.groups, p.strips - strip);
        p.first_row = static_cast<int>(strip) * rows;
        p.total = static_cast<uint32_t>(count * p.groups);
        kernel<<<(p.total - 1) / kThreads + 1, kThreads, 0, stream>>>(x + plane * H * W, y + plane * p.OH * p.OW, p,
                                                                      vec_out);
        first += count;
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return msda::note_cuda_error(e);
    msda::count_launches(launches);
    return MSDA_OK;
}

}  // namespace

extern "C" {

int addrelu_sm100_forward(void* x, const void* y, size_t n, int dtype, void* stream) {
    return dispatch_pointwise<false>(x, y, x, n, dtype, stream);
}

int addrelu_sm100_forward_out(const void* x, const void* y, void* out, size_t n, int dtype,
                              void* stream) {
    return dispatch_pointwise<false>(x, y, out, n, dtype, stream);
}

int addrelu_sm100_backward(const void* out, const void* grad_out, void* grad_in, size_t n,
                           int dtype, void* stream) {
    return dispatch_pointwise<true>(out, grad_out, grad_in, n, dtype, stream);
}

int maxpool_sm100_forward(const void* x, void* y, int N, int C, int H, int W, int dtype,
                          void* stream) {
    if (x == nullptr || y == nullptr) return MSDA_ERR_NULL;
    if (N < 0 || C < 0 || H < 0 || W < 0) return MSDA_ERR_DIMS;
    const size_t planes = static_cast<size_t>(N) * C;
    if (planes * H * W == 0) return MSDA_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    switch (dtype) {
        case MSDA_F32:
            return launch_maxpool(static_cast<const float*>(x), static_cast<float*>(y), planes, H, W, s);
        case MSDA_F16:
            return launch_maxpool(static_cast<const __half*>(x), static_cast<__half*>(y), planes, H, W, s);
        case MSDA_BF16:
            return launch_maxpool(static_cast<const __nv_bfloat16*>(x), static_cast<__nv_bfloat16*>(y), planes, H, W, s);
        default: return MSDA_ERR_DTYPE;
    }
}

}  // extern "C"
