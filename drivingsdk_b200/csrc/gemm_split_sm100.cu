// C[M, N] = sum_k A[m, k] * B[n, k] on the sm_100a tensor cores, operands as fp16 pairs
// (gemm_split.h), fp32 accumulation in tensor memory.
//
// Persistent, one CTA per SM, work item = 128 x BN tile of C over one part of K; K in stages of 32:
//   warp 0       producer: one TMA load per operand and stage brings both planes
//   warp 1       MMA: per 16 k three tcgen05.mma.kind::f16 (lo*hi, hi*lo, hi*hi) into one of two
//                accumulators
//   warps 2..5   epilogue of the finished accumulator: scales back, bias, stores (reductions when
//                K is cut across items); overlaps the products of the next item
// Nothing touches a stage between TMA and MMA, which is what the TF32 kernel spends its shared
// memory bandwidth on: per k of a 128 x 256 tile 1.5 KB come in and 2.3 KB go to the tensor core.
// The three products of the operator's test shape (M, N, K = 26100, 512, 4608 in the three orders)
// take 775 us together, 1.43 PFLOP/s of fp16 products; the TF32 kernel takes 1813 us.
// Every barrier wait is bounded; a time-out sets the status word, ends the CTA's work and drains
// what it issued, as in gemm_tc_sm100.cu.
#include <cuda_fp16.h>

#include "gemm_common.cuh"
#include "gemm_split.h"
#include "msda_launch.h"
#include "split_scale.cuh"

namespace msda {
namespace {

constexpr int BM = 128;
constexpr int BK = 32;
constexpr int kSplitThreads = 192;

template <int BN>
struct SplitTile {
    static constexpr int kPlaneA = BM * BK * 2;       // bytes of one plane of a stage
    static constexpr int kPlaneB = BN * BK * 2;
    static constexpr int kStageBytes = 2 * (kPlaneA + kPlaneB);
    static constexpr int kFit = (192 * 1024) / kStageBytes;
    static constexpr int kStages = kFit > 8 ? 8 : kFit;
    static constexpr int kSmemBytes = kStages * kStageBytes + 256 + 1024;
};

__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, int c0, int c1, int c2,
                                            int c3, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
        : "memory");
}

// Row-contiguous fp16 tile: blocks of 64 rows, a block being BK lines (k) of 128 bytes, 128-byte
// swizzle over groups of eight lines.
__device__ __forceinline__ uint64_t operand_desc_rows(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>((BK * 128) >> 4) << 16;       // next 64 rows
    d |= static_cast<uint64_t>(1024 >> 4) << 32;             // next 8 k
    d |= 1ull << 46;
    d |= 2ull << 61;
    return d;
}

__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc,
                                        uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

struct SplitParams {
    float* C;
    long long ldc;
    const float* bias;
    SplitScale a_scale, b_scale;
    int M, N, K;
    int kb_per_split, n_splits;
    int n_tiles, total_tiles;
    int row_major;      // operands have the row index contiguous
    int reduce;
    int vec;            // 32-byte stores / 16-byte reductions are aligned
    RangeGate gate;
    int* status;
};

struct SplitItem {
    int m0, n0, kb_begin, num_kb, split;
};
template <int BN>
__device__ __forceinline__ SplitItem split_item(const SplitParams& p, int w) {
    SplitItem it;
    it.split = w / p.total_tiles;
    const int tile = w - it.split * p.total_tiles;
    it.m0 = (tile / p.n_tiles) * BM;
    it.n0 = (tile % p.n_tiles) * BN;
    it.kb_begin = it.split * p.kb_per_split;
    it.num_kb = min((p.K + BK - 1) / BK, it.kb_begin + p.kb_per_split) - it.kb_begin;
    return it;
}

template <int BN>
__global__ void __launch_bounds__(kSplitThreads, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                  const __grid_constant__ SplitParams p) {
    if (!gate_open(p.gate)) return;
    using T = SplitTile<BN>;
    constexpr int kStages = T::kStages;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base_u32 = smem_u32(smem_raw);
    uint8_t* tiles = smem_raw + ((1024u - (base_u32 & 1023u)) & 1023u);
    uint64_t* bars = reinterpret_cast<uint64_t*>(tiles + kStages * T::kStageBytes);
    uint64_t* full = bars;                          // TMA landed
    uint64_t* empty = bars + kStages;               // the MMAs that read the stage have finished
    uint64_t* accum_full = bars + 2 * kStages;      // [2]
    uint64_t* accum_empty = bars + 2 * kStages + 2; // [2]
    uint64_t* drained = bars + 2 * kStages + 4;     // abort path only
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 5);
    volatile uint32_t* abort_flag = tmem_slot + 1;
    static_assert((2 * kStages + 5) * 8 + 8 <= 256, "barrier area");

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int total_items = p.total_tiles * p.n_splits;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&accum_full[a], 1);
            mbar_init(&accum_empty[a], 4);
        }
        mbar_init(drained, 1);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_slot)),
                     "r"(static_cast<uint32_t>(2 * BN))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    auto give_up = [&]() {
        atomicOr(p.status, kStatusGemmTimeout);
        *abort_flag = 1;
    };

    if (warp == 0) {
        // ---------------- producer ----------------
        if (lane == 0) {
            uint32_t it = 0;
            for (int w = blockIdx.x; w < total_items && !*abort_flag; w += gridDim.x) {
                const SplitItem wi = split_item<BN>(p, w);
                for (int i = 0; i < wi.num_kb && !*abort_flag; ++i, ++it) {
                    const int s = it % kStages;
                    if (!gemm_wait(&empty[s], ((it / kStages) & 1u) ^ 1u)) {
                        give_up();
                        break;
                    }
                    uint8_t* st = tiles + s * T::kStageBytes;
                    mbar_expect_tx(&full[s], T::kStageBytes);
                    const int k0 = (wi.kb_begin + i) * BK;
                    if (p.row_major) {
                        tma_load_4d(st, &map_a, 0, k0, wi.m0 / 64, 0, &full[s]);
                        tma_load_4d(st + 2 * T::kPlaneA, &map_b, 0, k0, wi.n0 / 64, 0, &full[s]);
                    } else {
                        tma_load_3d(st, &map_a, k0, wi.m0, 0, &full[s]);
                        tma_load_3d(st + 2 * T::kPlaneA, &map_b, k0, wi.n0, 0, &full[s]);
                    }
                }
            }
            // let the copies that were issued land before the CTA goes away, whoever gave up
            const uint32_t first = it > static_cast<uint32_t>(kStages) ? it - kStages : 0u;
            for (uint32_t j = first; j < it; ++j) gemm_wait(&full[j % kStages], (j / kStages) & 1u);
        }
    } else if (warp == 1) {
        // ---------------- MMA issue ----------------
        if (lane == 0) {
            // fp16 x fp16 -> fp32, M = 128, N = BN; both operands k-major or both row-contiguous
            const uint32_t idesc = (1u << 4) | (p.row_major ? (3u << 15) : 0u) |
                                   (static_cast<uint32_t>(BN >> 3) << 17) |
                                   (static_cast<uint32_t>(BM >> 4) << 24);
            uint32_t it = 0, item = 0;
            bool ok = true;
            for (int w = blockIdx.x; w < total_items && ok; w += gridDim.x, ++item) {
                const SplitItem wi = split_item<BN>(p, w);
                const uint32_t acc = item & 1u;
                const uint32_t tmem_d = tmem_base + acc * BN;
                if (*abort_flag || !gemm_wait(&accum_empty[acc], ((item >> 1) & 1u) ^ 1u)) {
                    give_up();
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int i = 0; i < wi.num_kb; ++i, ++it) {
                    const int s = it % kStages;
                    if (*abort_flag || !gemm_wait(&full[s], (it / kStages) & 1u)) {
                        give_up();
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t a_hi = smem_u32(tiles + s * T::kStageBytes);
                    const uint32_t a_lo = a_hi + T::kPlaneA;
                    const uint32_t b_hi = a_lo + T::kPlaneA;
                    const uint32_t b_lo = b_hi + T::kPlaneB;
#pragma unroll
                    for (int kk = 0; kk < BK / 16; ++kk) {
                        uint64_t dah, dal, dbh, dbl;
                        if (p.row_major) {
                            const uint32_t off = kk * 2048;   // 16 k
                            dah = operand_desc_rows(a_hi + off);
                            dal = operand_desc_rows(a_lo + off);
                            dbh = operand_desc_rows(b_hi + off);
                            dbl = operand_desc_rows(b_lo + off);
                        } else {
                            const uint32_t off = kk * 32;     // 16 fp16 values along k
                            dah = operand_desc<BK * 2>(a_hi + off);
                            dal = operand_desc<BK * 2>(a_lo + off);
                            dbh = operand_desc<BK * 2>(b_hi + off);
                            dbl = operand_desc<BK * 2>(b_lo + off);
                        }
                        mma_f16(tmem_d, dal, dbh, idesc, (i > 0 || kk > 0) ? 1u : 0u);
                        mma_f16(tmem_d, dah, dbl, idesc, 1u);
                        mma_f16(tmem_d, dah, dbh, idesc, 1u);
                    }
                    mma_commit(&empty[s]);
                }
                if (ok) mma_commit(&accum_full[acc]);
            }
            if (!ok || *abort_flag) {
                // the MMAs already issued still write tensor memory and read the stages
                mma_commit(drained);
                gemm_wait(drained, 0u);
            }
        }
    } else {
        // ---------------- epilogue ----------------
        const int q = warp & 3;                       // tensor-memory lane quarter of this warp
        uint32_t item = 0;
        for (int w = blockIdx.x; w < total_items; w += gridDim.x, ++item) {
            const SplitItem wi = split_item<BN>(p, w);
            const uint32_t acc = item & 1u;
            const int m = wi.m0 + 32 * q + lane;
            const float a_back = m < p.M ? exp2_int(-split_exponent(p.a_scale, m)) : 0.f;
            if (*abort_flag || !gemm_wait(&accum_full[acc], (item >> 1) & 1u)) {
                if (lane == 0) give_up();
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
            for (int c = 0; c < BN / 32; ++c) {
                const int n_first = wi.n0 + c * 32;
                if (n_first >= p.N) break;
                // this lane's column: its scale and bias reach the others by shuffle
                const int mine = min(n_first + lane, p.N - 1);
                const float b_back = exp2_int(-split_exponent(p.b_scale, mine));
                const float bias = (p.bias != nullptr && wi.split == 0) ? p.bias[mine] : 0.f;
                uint32_t r[32];
                tmem_load_32(tmem_base + (static_cast<uint32_t>(32 * q) << 16) + acc * BN + c * 32, r);
                float* row = p.C + static_cast<long long>(m) * p.ldc + n_first;
#pragma unroll
                for (int j = 0; j < 32; j += 8) {
                    float v[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e)
                        v[e] = fmaf(__uint_as_float(r[j + e]) * a_back,
                                    __shfl_sync(0xffffffffu, b_back, j + e),
                                    __shfl_sync(0xffffffffu, bias, j + e));
                    if (m >= p.M) continue;
                    if (p.vec && n_first + j + 7 < p.N) {
                        if (p.reduce) {
                            red_add_f32x4(row + j, v[0], v[1], v[2], v[3]);
                            red_add_f32x4(row + j + 4, v[4], v[5], v[6], v[7]);
                        } else {
                            // a whole 32-byte sector per lane
                            asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(row + j),
                                         "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]),
                                         "f"(v[5]), "f"(v[6]), "f"(v[7])
                                         : "memory");
                        }
                    } else {
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            if (n_first + j + e < p.N) {
                                if (p.reduce) atomicAdd(row + j + e, v[e]);
                                else row[j + e] = v[e];
                            }
                        }
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&accum_empty[acc]);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                     "r"(static_cast<uint32_t>(2 * BN))
                     : "memory");
    }
}

// Both planes of an operand in one map. k contiguous: [2][rows][K], boxes of 32 k x box_rows x 2.
// Row index contiguous: [2][rows / 64][K][64], boxes of 64 x 32 k x (box_rows / 64) x 2; the last
// block may reach past the last row, whose products are not stored.
cudaError_t make_split_map(CUtensorMap* map, const SplitOperand& o, int rows, int K, int box_rows) {
    EncodeTiledFn fn = nullptr;
    cudaError_t e = encode_fn(&fn);
    if (e != cudaSuccess) return e;
    void* base = const_cast<uint16_t*>(o.hi);
    const cuuint64_t plane = static_cast<cuuint64_t>(o.plane) * 2;
    const cuuint32_t unit[4] = {1, 1, 1, 1};
    CUresult r;
    if (o.k_stride == 1) {
        const cuuint64_t dims[3] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(rows), 2};
        const cuuint64_t strides[2] = {static_cast<cuuint64_t>(o.row_stride) * 2, plane};
        const cuuint32_t box[3] = {BK, static_cast<cuuint32_t>(box_rows), 2};
        r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, base, dims, strides, box, unit,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    } else {
        const cuuint64_t dims[4] = {64, static_cast<cuuint64_t>(K),
                                    static_cast<cuuint64_t>((rows + 63) / 64), 2};
        const cuuint64_t strides[3] = {static_cast<cuuint64_t>(o.k_stride) * 2, 128, plane};
        const cuuint32_t box[4] = {64, BK, static_cast<cuuint32_t>(box_rows / 64), 2};
        r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, base, dims, strides, box, unit,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    }
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

template <int BN>
cudaError_t launch_split(const SplitOperand& A, const SplitOperand& B, SplitParams p, int splits,
                         cudaStream_t stream) {
    int resident = 0;   // one CTA per SM; the call sets the shared-memory limit
    cudaError_t e = resident_ctas(reinterpret_cast<const void*>(gemm_split_kernel<BN>), kSplitThreads,
                                  SplitTile<BN>::kSmemBytes, &resident);
    if (e != cudaSuccess) return e;
    CUtensorMap map_a, map_b;
    e = make_split_map(&map_a, A, p.M, p.K, BM);
    if (e != cudaSuccess) return e;
    e = make_split_map(&map_b, B, p.N, p.K, BN);
    if (e != cudaSuccess) return e;
    const int kb_total = (p.K + BK - 1) / BK;
    if (splits < 1) splits = 1;
    if (splits > kb_total) splits = kb_total;
    p.kb_per_split = (kb_total + splits - 1) / splits;
    p.n_splits = (kb_total + p.kb_per_split - 1) / p.kb_per_split;   // no part is empty
    p.reduce = splits > 1 ? 1 : 0;
    p.n_tiles = (p.N + BN - 1) / BN;
    const long long tiles = static_cast<long long>((p.M + BM - 1) / BM) * p.n_tiles;
    const long long items = tiles * p.n_splits;
    if (items >= (1ll << 31)) return cudaErrorInvalidValue;
    p.total_tiles = static_cast<int>(tiles);
    int sms = 0;
    if (device_facts(&sms, nullptr) != 0) return cudaErrorInvalidDevice;
    gemm_split_kernel<BN><<<static_cast<unsigned>(items < sms ? items : sms), kSplitThreads,
                            SplitTile<BN>::kSmemBytes, stream>>>(map_a, map_b, p);
    return cudaGetLastError();
}

}  // namespace

cudaError_t gemm_split(const SplitOperand& A, const SplitOperand& B, float* C, long long ldc,
                       const float* bias, int M, int N, int K, int splits, const RangeGate& gate,
                       int* status_word, cudaStream_t stream) {
    if (M <= 0 || N <= 0 || K <= 0 || status_word == nullptr) return cudaErrorInvalidValue;
    const bool rows = A.k_stride != 1;
    for (const SplitOperand* o : {&A, &B}) {
        const long long step = rows ? o->k_stride : o->row_stride;
        if ((rows ? o->row_stride : o->k_stride) != 1 || step % 8 != 0 || o->plane % 8 != 0 ||
            reinterpret_cast<uintptr_t>(o->hi) % 16 != 0)
            return cudaErrorInvalidValue;
    }
    SplitParams p{};
    p.C = C;
    p.ldc = ldc;
    p.bias = bias;
    p.a_scale = A.scale;
    p.b_scale = B.scale;
    p.M = M;
    p.N = N;
    p.K = K;
    p.row_major = rows ? 1 : 0;
    p.vec = (ldc % 8 == 0 && reinterpret_cast<uintptr_t>(C) % 32 == 0) ? 1 : 0;
    p.gate = gate;
    p.status = status_word;
    if (N > 192) return launch_split<256>(A, B, p, splits, stream);
    if (N > 96) return launch_split<128>(A, B, p, splits, stream);
    return launch_split<64>(A, B, p, splits, stream);
}

}  // namespace msda
