// Prefill GEMM (m > 8): Y[m,n] = X[m,k] . W[n,k]^T on the 5th-generation tensor cores.
//
// CQ_ACT_F16 numerics: activations rounded to f16, weights dequantized (exactly, in f32) and
// rounded once to f16, products exact, accumulation in f32 inside the tensor core.  Against
// candy's CPU path (f32 activations, conv.go:373-389) this differs by the two f16 roundings:
// ~3e-4 of max|y| on the benchmark's distributions, inside the 1e-3 bar.  Why not int8 MMAs:
// each 32-block carries its own scale on BOTH operands (d_w[n,b] * d_x[m,b]), a rank-1 factor per
// block that no single int8 operand can absorb, so an int8 design has to drain the accumulator
// every 32 values of k and rescale on CUDA cores -- about 4 CUDA-core instructions per 32 MACs,
// which caps it near one eighth of the int8 pipe, below this f16 kernel, and single-slice int8
// activations miss the 1e-3 bar against the CPU path (5.8e-3) anyway.
//
// Two steps.  (1) streaming conversion kernels write f16 copies of X [m,k] and W [n,k] into
// context scratch (HBM-bound: 18/34 B in, 64 B out per block).  (2) gemm_f16_tn_kernel: one CTA
// per 128 x 256 (or, for m <= 64, 128 x 64) output tile; a producer lane feeds a shared-memory ring with TMA tensor
// loads (128-byte swizzle, K-major tiles of 64 values); one lane issues tcgen05.mma
// (cta_group::1, kind::f16, M=128, N=256, K=16 x 4 per stage) into a 256-column f32 accumulator
// in tensor memory; tcgen05.commit hands stages back to the producer and, at the end, the
// accumulator to four epilogue warps that read it with tcgen05.ld and store f32 rows.
// Every mbarrier wait is bounded; a give-up sets the context's error word and the CTA still
// reaches the final barrier and frees its tensor memory.
#include "common.cuh"
#include "tcgen05.cuh"

namespace {

constexpr int BM = 128, BK = 64;
constexpr int A_BYTES = BM * BK * 2;  // 16 KiB
constexpr int GEMM_THREADS = 192;     // warp 0: TMA, warp 1: MMA + TMEM, warps 2-5: epilogue
// Two tile shapes: 128 x 256 (4 stages) for wide batches, 128 x 64 (8 stages) for batches of at
// most 64 rows, where the number of n-tiles is what fills the SMs.
template <int BN>
struct GemmCfg {
    static constexpr int kStages = BN >= 256 ? 4 : 8;
    static constexpr int kBBytes = BN * BK * 2;
    static constexpr int kTmemCols = BN < 32 ? 32 : BN;
    static constexpr size_t kSmem = (size_t)kStages * (A_BYTES + kBBytes) + 1024 /* alignment slack */ + 256 /* barriers */;
};

// ---- f16 conversion kernels -------------------------------------------------------------
// CTA `cta` of `ctas` of X [m, k] f32 -> f16: 16 bytes in where X allows it.
__device__ __forceinline__ void x_part_to_f16(const float *__restrict__ x, int64_t m, int64_t k, int64_t ldx, __half *__restrict__ out, unsigned cta,
                                              unsigned ctas) {
    const int64_t total = m * (k / 4);
    const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0 && ldx % 4 == 0;
    for (int64_t i = (int64_t)cta * blockDim.x + threadIdx.x; i < total; i += (int64_t)ctas * blockDim.x) {
        const int64_t row = i / (k / 4), c4 = i - row * (k / 4);
        const float *src = x + row * ldx + c4 * 4;
        const float4 t = vec ? *reinterpret_cast<const float4 *>(src) : make_float4(src[0], src[1], src[2], src[3]);
        __half2 a = __floats2half2_rn(t.x, t.y), b = __floats2half2_rn(t.z, t.w);
        uint2 v;
        v.x = *reinterpret_cast<uint32_t *>(&a);
        v.y = *reinterpret_cast<uint32_t *>(&b);
        *reinterpret_cast<uint2 *>(out + row * k + c4 * 4) = v;
    }
}
__global__ void __launch_bounds__(256) x_to_f16_kernel(const float *__restrict__ x, int64_t m, int64_t k, int64_t ldx, __half *__restrict__ out) {
    x_part_to_f16(x, m, k, ldx, out, blockIdx.x, gridDim.x);
}

// Eight bytes that start at any even address, as two words: the aligned words around them, shifted into place.
__device__ __forceinline__ void eight_bytes(const uint8_t *p, uint32_t &a, uint32_t &b) {
    const uint32_t odd = (uint32_t)(reinterpret_cast<uintptr_t>(p) & 2);
    const uint32_t *q = reinterpret_cast<const uint32_t *>(p - odd);
    const uint32_t v0 = q[0], v1 = q[1], v2 = odd ? q[2] : 0u;
    a = __funnelshift_r(v0, v1, 8 * odd);
    b = __funnelshift_r(v1, v2, 8 * odd);
}

// Both f16 copies in one launch: the first x_ctas CTAs convert X, the others W.
// W: one thread converts 8 consecutive values of a block (one 16-byte store).  The f32 value
// d*(q-8) (or d*q) is exact, so the only rounding is f32 -> f16, round-to-nearest-even.
// Bound: HBM (0.56 / 1.06 bytes in, 2 out per weight).  One launch that the GEMM may overlap instead of two that it may
// not: n 11008, k 4096, 2048 rows of Q8_0 183 -> 172 us a call, of Q4_0 in the split order 183 -> 170.
template <int QT, int ORDER>
__global__ void __launch_bounds__(256) operands_to_f16_kernel(const uint8_t *__restrict__ blocks, int64_t nblocks, __half *__restrict__ out, unsigned x_ctas,
                                                            const float *__restrict__ x, int64_t m, int64_t k, int64_t ldx, __half *__restrict__ x_out) {
    pdl_launch_dependents();  // the GEMM sets itself up meanwhile
    if (blockIdx.x < x_ctas) {
        x_part_to_f16(x, m, k, ldx, x_out, blockIdx.x, x_ctas);
        return;
    }
    const int64_t total = nblocks * 4;
    const int64_t step = (int64_t)(gridDim.x - x_ctas) * blockDim.x;
    for (int64_t idx = (int64_t)(blockIdx.x - x_ctas) * blockDim.x + threadIdx.x; idx < total; idx += step) {
        const int64_t blk = idx >> 2;
        const int p = (int)(idx & 3);  // values 8p .. 8p+7
        float v[8];
        const uint8_t *b = blocks + blk * (QT == CQ_Q4_0 ? kQ4Bytes : kQ8Bytes);
        const float d = __half2float(__ushort_as_half(*reinterpret_cast<const unsigned short *>(b)));
        if (QT == CQ_Q4_0) {
            if (ORDER == CQ_ORDER_GO_INTERLEAVED) {
                const uint8_t *qs = b + 2 + 4 * p;  // bytes 4p..4p+3 -> values 8p..8p+7
                const uint32_t four = *reinterpret_cast<const unsigned short *>(qs) |
                                      ((uint32_t) * reinterpret_cast<const unsigned short *>(qs + 2) << 16);
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = d * (float)((int)((four >> (4 * i)) & 0xF) - 8);
            } else {
                uint32_t w[2];  // values 8p .. = low (p < 2) or high nibbles of 8 bytes
                eight_bytes(b + 2 + 8 * (p & 1), w[0], w[1]);
                const int sh = (p >= 2) ? 4 : 0;
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = d * (float)((int)((w[i >> 2] >> (8 * (i & 3) + sh)) & 0xF) - 8);
            }
        } else {
            uint32_t w[2];
            eight_bytes(b + 2 + 8 * p, w[0], w[1]);
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = d * (float)(int)(signed char)((w[i >> 2] >> (8 * (i & 3))) & 0xFF);
        }
        __half2 h[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
        *reinterpret_cast<uint4 *>(out + idx * 8) = *reinterpret_cast<uint4 *>(h);
    }
}

template <int BN>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
    gemm_f16_tn_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, float *__restrict__ y, int M,
                       int N, int K, int64_t ldy, int *err) {
    constexpr int STAGES = GemmCfg<BN>::kStages, B_BYTES = GemmCfg<BN>::kBBytes, TMEM_COLS = GemmCfg<BN>::kTmemCols;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *smA = smem;                              // [STAGES][A_BYTES]
    uint8_t *smB = smem + (size_t)STAGES * A_BYTES;   // [STAGES][B_BYTES]
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + (size_t)STAGES * (A_BYTES + B_BYTES));
    uint64_t *full = bars, *empty = bars + STAGES, *acc_full = bars + 2 * STAGES;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * STAGES + 1);

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    // m-tiles vary fastest across the grid: a wave of CTAs then shares a handful of B tiles (and all
    // of A), so the f16 weight copy crosses HBM about once instead of once per few m-tiles.
    const int tile_m = blockIdx.x, tile_n = blockIdx.y;
    const int nk = (K + BK - 1) / BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(&full[s]), 1);
            mbar_init(smem_u32(&empty[s]), 1);
        }
        mbar_init(smem_u32(acc_full), 1);
        fence_mbar_init();
        fence_proxy_async();
    }
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            int issued = 0;
            for (int kb = 0; kb < nk; ++kb) {
                const int s = kb % STAGES;
                if (kb >= STAGES && !mbar_wait_bounded(smem_u32(&empty[s]), ((kb / STAGES) - 1) & 1)) {
                    atomicExch(err, kDevErrEmptyWait);
                    break;
                }
                mbar_expect_tx(smem_u32(&full[s]), A_BYTES + B_BYTES);
                tma_load_2d(smem_u32(smA + (size_t)s * A_BYTES), &tmA, kb * BK, tile_m * BM, smem_u32(&full[s]));
                tma_load_2d(smem_u32(smB + (size_t)s * B_BYTES), &tmB, kb * BK, tile_n * BN, smem_u32(&full[s]));
                issued = kb + 1;
            }
            // never leave with copies in flight into this CTA's shared memory
            const int first = issued > STAGES ? issued - STAGES : 0;
            for (int kb = first; kb < issued; ++kb)
                if (!mbar_wait_bounded(smem_u32(&full[kb % STAGES]), (kb / STAGES) & 1)) {
                    atomicExch(err, kDevErrDrain);
                    break;
                }
        }
    } else if (warp == 1) {
        {  // the whole warp runs the loop, one lane issues (n 11008, k 4096, 64 rows of Q4_1: 77 -> 66 us a call)
            constexpr uint32_t idesc = idesc_f16(BM, BN);
            for (int kb = 0; kb < nk; ++kb) {
                const int s = kb % STAGES;
                if (!__all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&full[s]), (kb / STAGES) & 1))) {
                    if (lane == 0) atomicExch(err, kDevErrFullWait);
                    break;
                }
                tc_fence_after();
                const uint32_t a0 = smem_u32(smA + (size_t)s * A_BYTES), b0 = smem_u32(smB + (size_t)s * B_BYTES);
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k)  // 16 values of k = 32 bytes inside the 128-byte swizzled row
                        tc_mma_f16(tmem_base, smem_desc_k128(a0 + 32 * k), smem_desc_k128(b0 + 32 * k), idesc, (kb | k) != 0);
                    tc_commit(smem_u32(&empty[s]));  // arrives when these MMAs have finished reading the stage
                }
                __syncwarp();
            }
            if (elect_one()) tc_commit(smem_u32(acc_full));  // arrives when every MMA issued so far has completed
        }
    } else {
        // epilogue warps 2..5: warp w may touch TMEM lanes 32*(w%4) .. +31 only
        const int q = warp & 3;
        if (mbar_wait_bounded(smem_u32(acc_full), 0)) {
            tc_fence_after();
            const int64_t row = (int64_t)tile_m * BM + q * 32 + lane;
            const int col0 = tile_n * BN;
#pragma unroll 1
            for (int c = 0; c < BN / 32; ++c) {
                uint32_t r[32];
                tmem_ld32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(c * 32), r);
                const int col = col0 + c * 32;
                if (row < M) {
                    float *dst = y + row * ldy + col;
                    if (col + 32 <= N && ((reinterpret_cast<uintptr_t>(dst) & 15) == 0)) {
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            reinterpret_cast<float4 *>(dst)[i] = make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]),
                                                                             __uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3]));
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (col + i < N) dst[i] = __uint_as_float(r[i]);
                    }
                }
            }
        } else if (lane == 0) {
            atomicExch(err, kDevErrMma);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

// Persistent variant of the 128 x 256 kernel: one CTA per SM walks tiles t = blockIdx.x, +gridDim.x, ...
// (m-tiles fastest).  The shared-memory ring keeps running across tile boundaries and the
// accumulator is double-buffered in tensor memory (2 x 256 columns), so the epilogue of tile i
// overlaps the MMAs of tile i+1 and no tile pays the pipeline fill again.
__global__ void __launch_bounds__(GEMM_THREADS, 1)
    gemm_f16_tn_persistent_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, float *__restrict__ y,
                                  int M, int N, int K, int64_t ldy, int *err) {
    constexpr int BN = 256;
    constexpr int STAGES = GemmCfg<BN>::kStages, B_BYTES = GemmCfg<BN>::kBBytes;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *smA = smem;
    uint8_t *smB = smem + (size_t)STAGES * A_BYTES;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + (size_t)STAGES * (A_BYTES + B_BYTES));
    uint64_t *full = bars, *empty = bars + STAGES, *acc_full = bars + 2 * STAGES, *acc_empty = bars + 2 * STAGES + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * STAGES + 4);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int mt = (M + BM - 1) / BM, nt = (N + BN - 1) / BN;
    const int ntiles = mt * nt;
    const int nk = (K + BK - 1) / BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(smem_u32(&full[s]), 1);
            mbar_init(smem_u32(&empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&acc_full[b]), 1);
            mbar_init(smem_u32(&acc_empty[b]), 4);  // one arrival per epilogue warp
        }
        fence_mbar_init();
        fence_proxy_async();
    }
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            int it = 0;  // k-blocks issued so far, across tiles
            bool ok = true;
            for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
                const int tile_m = t % mt, tile_n = t / mt;
                for (int kb = 0; kb < nk; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (it >= STAGES && !mbar_wait_bounded(smem_u32(&empty[s]), ((it / STAGES) - 1) & 1)) {
                        atomicExch(err, kDevErrEmptyWait);
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(smem_u32(&full[s]), A_BYTES + B_BYTES);
                    tma_load_2d(smem_u32(smA + (size_t)s * A_BYTES), &tmA, kb * BK, tile_m * BM, smem_u32(&full[s]));
                    tma_load_2d(smem_u32(smB + (size_t)s * B_BYTES), &tmB, kb * BK, tile_n * BN, smem_u32(&full[s]));
                }
            }
            // never leave with copies in flight into this CTA's shared memory
            const int first = it > STAGES ? it - STAGES : 0;
            for (int i = first; i < it; ++i)
                if (!mbar_wait_bounded(smem_u32(&full[i % STAGES]), (i / STAGES) & 1)) {
                    atomicExch(err, kDevErrDrain);
                    break;
                }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = idesc_f16(BM, BN);
            int it = 0, ti = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x, ++ti) {
                const int buf = ti & 1;
                if (ti >= 2 && !mbar_wait_bounded(smem_u32(&acc_empty[buf]), ((ti >> 1) - 1) & 1)) {  // epilogue done with this buffer
                    atomicExch(err, kDevErrMma);
                    break;
                }
                tc_fence_after();
                const uint32_t acc = tmem_base + (uint32_t)(buf * BN);
                for (int kb = 0; kb < nk; ++kb, ++it) {
                    const int s = it % STAGES;
                    if (!mbar_wait_bounded(smem_u32(&full[s]), (it / STAGES) & 1)) {
                        atomicExch(err, kDevErrFullWait);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a0 = smem_u32(smA + (size_t)s * A_BYTES), b0 = smem_u32(smB + (size_t)s * B_BYTES);
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k)
                        tc_mma_f16(acc, smem_desc_k128(a0 + 32 * k), smem_desc_k128(b0 + 32 * k), idesc, (kb | k) != 0);
                    tc_commit(smem_u32(&empty[s]));
                }
                tc_commit(smem_u32(&acc_full[buf]));
            }
        }
    } else {
        const int q = warp & 3;
        int ti = 0;
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++ti) {
            const int buf = ti & 1;
            const int tile_m = t % mt, tile_n = t / mt;
            if (!mbar_wait_bounded(smem_u32(&acc_full[buf]), (ti >> 1) & 1)) {
                if (lane == 0) atomicExch(err, kDevErrMma);
                break;
            }
            tc_fence_after();
            const int64_t row = (int64_t)tile_m * BM + q * 32 + lane;
            const int col0 = tile_n * BN;
#pragma unroll 1
            for (int c = 0; c < BN / 32; ++c) {
                uint32_t r[32];
                tmem_ld32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * BN + c * 32), r);
                const int col = col0 + c * 32;
                if (row < M) {
                    float *dst = y + row * ldy + col;
                    if (col + 32 <= N && ((reinterpret_cast<uintptr_t>(dst) & 15) == 0)) {
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            reinterpret_cast<float4 *>(dst)[i] = make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]),
                                                                             __uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3]));
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (col + i < N) dst[i] = __uint_as_float(r[i]);
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&acc_empty[buf]));  // this warp's quarter of the buffer is free
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, 512);
}


// ---- CTA pairs: one 256 x 256 output tile per two SMs (cta_group::2) -----------------------------------
// The persistent kernel above is bound by shared-memory bandwidth, not by the tensor pipe: per K = 16 step a
// 128 x 256 MMA reads 4 KB of A and 8 KB of B from the CTA's shared memory, 96 bytes per clock at the pipe's
// rate, next to the TMA writes of the same bytes.  With cta_group::2 the two CTAs of a cluster (the two SMs
// of a TPC) issue ONE MMA of M = 256: each CTA supplies its own 128 rows of A and HALF of the B tile (128 of
// the 256 weight rows) from its own shared memory and keeps the 128 x 256 accumulators of its rows in its own
// tensor memory, so each SM stages and reads 8 KB per step instead of 12 for the same work.
// Protocol (every barrier wait bounded): both CTAs' producer lanes issue their TMA loads with the LEADER's
// (cluster rank 0) full barrier as the completion barrier; the leader's producer arms it with the byte count of
// both; the leader's MMA lane waits on it, issues the pair's MMAs and commits to the empty barrier of BOTH CTAs
// (and, at the end of a tile, to both accumulator-full barriers); the epilogue warps of both CTAs drain their own
// tensor memory and arrive on the leader's accumulator-empty barrier.  Cluster barriers after the barrier set-up
// and before the end keep either CTA from touching the other's barriers too early or leaving too soon.
constexpr int P2_STAGES = 6;
constexpr int P2_BH_BYTES = 128 * BK * 2;  // this CTA's half of the B tile: 16 KB
constexpr int P2_STAGE_BYTES = A_BYTES + P2_BH_BYTES;
constexpr size_t P2_SMEM = (size_t)P2_STAGES * P2_STAGE_BYTES + 1024 + 256;

__global__ void __launch_bounds__(GEMM_THREADS, 1)
    gemm_f16_tn_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, float *__restrict__ y, int M,
                            int N, int K, int64_t ldy, int *err) {
    constexpr int BN = 256;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *smA = smem;                                    // [P2_STAGES][A_BYTES]
    uint8_t *smB = smem + (size_t)P2_STAGES * A_BYTES;      // [P2_STAGES][P2_BH_BYTES]
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + (size_t)P2_STAGES * P2_STAGE_BYTES);
    uint64_t *full = bars, *empty = bars + P2_STAGES, *acc_full = bars + 2 * P2_STAGES, *acc_empty = bars + 2 * P2_STAGES + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * P2_STAGES + 4);

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
    const int mt = (M + 255) / 256, nt = (N + BN - 1) / BN;
    const int ntiles = mt * nt;
    const int nk = (K + BK - 1) / BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < P2_STAGES; ++s) {
            mbar_init(smem_u32(&full[s]), 1);
            mbar_init(smem_u32(&empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&acc_full[b]), 1);
            mbar_init(smem_u32(&acc_empty[b]), 8);  // four epilogue warps of each CTA
        }
        fence_mbar_init();
        fence_proxy_async();
    }
    __syncthreads();
    cluster_sync_all();  // the peer's barriers exist before anything of this CTA can signal them
    if (warp == 1) tmem_alloc_pair(smem_u32(tmem_slot), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            pdl_wait_prior();  // the f16 copies come from the kernel before
            int it = 0;
            bool ok = true;
            for (int t = pair; t < ntiles && ok; t += npairs) {
                const int tile_m = t % mt, tile_n = t / mt;
                for (int kb = 0; kb < nk; ++kb, ++it) {
                    const int s = it % P2_STAGES;
                    if (it >= P2_STAGES && !mbar_wait_bounded(smem_u32(&empty[s]), ((it / P2_STAGES) - 1) & 1)) {
                        atomicExch(err, kDevErrEmptyWait);
                        ok = false;
                        break;
                    }
                    const uint32_t lead_full = mapa_shared(smem_u32(&full[s]), 0);
                    if (rank == 0) mbar_expect_tx(smem_u32(&full[s]), 2 * P2_STAGE_BYTES);
                    tma_load_2d_pair(smem_u32(smA + (size_t)s * A_BYTES), &tmA, kb * BK, tile_m * 256 + (int)rank * 128, lead_full);
                    tma_load_2d_pair(smem_u32(smB + (size_t)s * P2_BH_BYTES), &tmB, kb * BK, tile_n * BN + (int)rank * 128, lead_full);
                }
            }
            if (rank == 0 && ok) {  // the leader's full barriers count the bytes of both CTAs: wait for the last ones
                const int first = it > P2_STAGES ? it - P2_STAGES : 0;
                for (int i = first; i < it; ++i)
                    if (!mbar_wait_bounded(smem_u32(&full[i % P2_STAGES]), (i / P2_STAGES) & 1)) {
                        atomicExch(err, kDevErrDrain);
                        break;
                    }
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {  // the whole warp runs the loop, one lane issues (n 11008, k 4096, 2048 rows of Q8_0: 187 -> 182 us a call)
            constexpr uint32_t idesc = idesc_f16(256, BN);
            int it = 0, ti = 0;
            bool ok = true;
            for (int t = pair; t < ntiles && ok; t += npairs, ++ti) {
                const int buf = ti & 1;
                if (ti >= 2 && !__all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&acc_empty[buf]), ((ti >> 1) - 1) & 1))) {
                    if (lane == 0) atomicExch(err, kDevErrMma);
                    break;
                }
                tc_fence_after();
                const uint32_t acc = tmem_base + (uint32_t)(buf * BN);
                for (int kb = 0; kb < nk; ++kb, ++it) {
                    const int s = it % P2_STAGES;
                    if (!__all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&full[s]), (it / P2_STAGES) & 1))) {
                        if (lane == 0) atomicExch(err, kDevErrFullWait);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a0 = smem_u32(smA + (size_t)s * A_BYTES), b0 = smem_u32(smB + (size_t)s * P2_BH_BYTES);
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < BK / 16; ++k)
                            tc_mma_f16_pair(acc, smem_desc_k128(a0 + 32 * k), smem_desc_k128(b0 + 32 * k), idesc, (kb | k) != 0);
                        tc_commit_pair(smem_u32(&empty[s]), 3);
                        if (kb == nk - 1) tc_commit_pair(smem_u32(&acc_full[buf]), 3);
                    }
                    __syncwarp();
                }
            }
        }
    } else {
        const int q = warp & 3;
        const uint32_t lead_acc_empty0 = mapa_shared(smem_u32(&acc_empty[0]), 0);
        int ti = 0;
        for (int t = pair; t < ntiles; t += npairs, ++ti) {
            const int buf = ti & 1;
            const int tile_m = t % mt, tile_n = t / mt;
            if (!mbar_wait_bounded(smem_u32(&acc_full[buf]), (ti >> 1) & 1)) {
                if (lane == 0) atomicExch(err, kDevErrMma);
                break;
            }
            tc_fence_after();
            const int64_t row = (int64_t)tile_m * 256 + (int)rank * 128 + q * 32 + lane;
            const int col0 = tile_n * BN;
#pragma unroll 1
            for (int c = 0; c < BN / 32; ++c) {
                uint32_t r[32];
                tmem_ld32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * BN + c * 32), r);
                const int col = col0 + c * 32;
                if (row < M) {
                    float *dst = y + row * ldy + col;
                    if (col + 32 <= N && ((reinterpret_cast<uintptr_t>(dst) & 15) == 0)) {
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            reinterpret_cast<float4 *>(dst)[i] = make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]),
                                                                             __uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3]));
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (col + i < N) dst[i] = __uint_as_float(r[i]);
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(lead_acc_empty0 + 8 * buf);  // this warp's quarter of this CTA's buffer is free
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // neither CTA leaves (or frees tensor memory) while the pair's MMAs may still use it
    if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
}

// ---- host side ----------------------------------------------------------------------------
// f16 [rows, k] row-major; box = 64 values of k x box_rows rows, 128-byte swizzle, zero fill outside.
bool make_map(CUtensorMap *map, const void *base, int64_t rows, int64_t k, int box_rows) {  // box_rows <= 256
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)k * 2};
    cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

cq_status launch_gemm(cq_ctx *ctx, int qtype, int order, int actmode, const float *x, int64_t m, int64_t k, int64_t ldx,
                      const void *w, int64_t n, float *y, int64_t ldy) {
    if (actmode == CQ_ACT_F32 && ctx->tune.gemv_variant == 0 && !ctx->tune.force_simple && (reinterpret_cast<uintptr_t>(x) & 15) == 0 && ldx % 4 == 0 &&
        gemv_f32_supported(qtype, w, x, y) && (cq_is_more_format(qtype) || cq_is_k_format(qtype) || !qgemm_i8_supported(qtype, k, w, x, ldx)))
        return launch_gemv_f32(ctx, qtype, order, x, m, k, ldx, w, n, y, ldy);
    if (actmode != CQ_ACT_F16) {
        // f32 / Q8_1 activation numerics for m > 8: the decode kernels, eight rows at a time
        // (weights are re-read once per eight rows; the tensor-core path is CQ_ACT_F16).
        for (int64_t r = 0; r < m; r += 8) {
            const int64_t rows = (m - r) < 8 ? (m - r) : 8;
            cq_status s = launch_gemv(ctx, qtype, order, actmode, x + r * ldx, rows, k, ldx, w, n, y + r * ldy, ldy);
            if (s != CQ_OK) return s;
        }
        return CQ_OK;
    }
    if ((reinterpret_cast<uintptr_t>(w) & 1) != 0 || (reinterpret_cast<uintptr_t>(x) & 3) != 0 || (reinterpret_cast<uintptr_t>(y) & 3) != 0)
        return cq_fail(ctx, CQ_ERR_INVALID_ARG, "gemm: misaligned pointer");
    if (m > 0x7FFFFFFF || n > 0x7FFFFFFF || k > 0x7FFFFFFF) return cq_fail(ctx, CQ_ERR_TOO_LARGE, "gemm: dimension beyond 2^31");
    // CTA pairs that dequantize raw blocks into tensor memory (gemm_pair_tmem.cu), n 11008 x k 4096, this kernel against the other
    // routes, us: 128 rows 23.8 / 28.6, 200 rows 34 / 56, 600 rows 64 / 80 (Q8_0: 74 / 84).  Its lines: past 1024 rows (Q8_0: 768)
    // the f16 copy of W, made once, costs less than dequantizing W again for every 128 rows (1024 rows 100 / 106, Q8_0 117 / 110;
    // 1300 rows 136 / 129, Q8_0 159 / 135); up to 32 rows the narrow kernel's loads are the quicker ones (16 rows 17.3 / 15.0), up
    // to 64 only on larger matrices (64 rows 20.1 / 21.1; 22016 x 4096 27.7 / 27.3, Q8_0 37.5 / 32.2).
    const int64_t items_per_sm = ((n + 255) / 256) * (k / 256) / ctx->sm_count;
    const bool pairs_win = m <= (qtype == CQ_Q4_0 ? 1024 : 768) && (m > 64 || (m > 32 && items_per_sm < 6));
    if (ctx->tune.gemm_variant == 0 && !ctx->tune.gemm_cache_weights && gemm_pair_tmem_supported(qtype, k, w) &&
        (ctx->tune.gemm_fused_dequant == 2 || (ctx->tune.gemm_fused_dequant == 1 && pairs_win)))
        return launch_gemm_pair_tmem(ctx, qtype, order, false, x, m, k, ldx, w, n, y, ldy);
    // narrow batches stream the raw blocks and dequantize into tensor memory: no f16 copy of W
    if (!cq_is_more_format(qtype) && !cq_is_k_format(qtype) && ctx->tune.gemm_variant != 3 && !ctx->tune.gemm_cache_weights && qgemm_dequant_tmem_supported(qtype, m, k, w))
        return launch_qgemm_dequant_tmem(ctx, qtype, order, x, m, k, ldx, w, n, y, ldy);
    const size_t x16_bytes = (((size_t)m * k * 2) + 1023) & ~size_t(1023);
    const size_t w16_bytes = (size_t)n * k * 2;
    // With gemm_cache_weights the f16 copy of a weight matrix is made once and kept (the caller
    // promises not to rewrite those blocks in place): later calls skip the conversion kernel.
    __half *w16 = nullptr;
    bool need_convert = true;
    const auto key = std::make_tuple(w, n, k, qtype * 2 + order);
    if (ctx->tune.gemm_cache_weights) {
        auto it = ctx->w16_cache.find(key);
        if (it != ctx->w16_cache.end()) {
            w16 = static_cast<__half *>(it->second);
            need_convert = false;
        } else {
            cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
            if (ctx->capturing || (cudaStreamIsCapturing(ctx->stream, &cap) == cudaSuccess && cap != cudaStreamCaptureStatusNone))
                return cq_fail(ctx, CQ_ERR_INVALID_ARG, "gemm: the cached f16 copy of this weight matrix does not exist yet and cannot be allocated during stream capture: run the call once before capturing");
            void *p = nullptr;
            CQ_CUDA(ctx, cq_device_malloc(ctx, &p, w16_bytes));
            ctx->w16_cache[key] = p;
            ctx->w16_cache_bytes += w16_bytes;
            w16 = static_cast<__half *>(p);
        }
    }
    cq_status s = cq_reserve_scratch(ctx, x16_bytes + (w16 ? 0 : w16_bytes));
    if (s != CQ_OK) return s;
    __half *x16 = static_cast<__half *>(ctx->scratch);
    if (!w16) w16 = reinterpret_cast<__half *>(static_cast<uint8_t *>(ctx->scratch) + x16_bytes);
    const unsigned cap = (unsigned)ctx->sm_count * 16;
    const int64_t xtotal = m * (k / 4);
    const unsigned xgrid = (unsigned)((xtotal + 255) / 256 < cap ? (xtotal + 255) / 256 : cap);
    bool chained = false;  // the kernel before the GEMM lets it start early
    if (need_convert && (qtype == CQ_Q4_0 || qtype == CQ_Q8_0)) {
        const int64_t nblocks = n * (k / kQK);
        const int64_t total = nblocks * 4;
        const unsigned grid = xgrid + (unsigned)((total + 255) / 256 < cap ? (total + 255) / 256 : cap);
        const uint8_t *wb = static_cast<const uint8_t *>(w);
        if (qtype == CQ_Q4_0 && order == CQ_ORDER_GO_INTERLEAVED) operands_to_f16_kernel<CQ_Q4_0, 0><<<grid, 256, 0, ctx->stream>>>(wb, nblocks, w16, xgrid, x, m, k, ldx, x16);
        else if (qtype == CQ_Q4_0) operands_to_f16_kernel<CQ_Q4_0, 1><<<grid, 256, 0, ctx->stream>>>(wb, nblocks, w16, xgrid, x, m, k, ldx, x16);
        else operands_to_f16_kernel<CQ_Q8_0, 0><<<grid, 256, 0, ctx->stream>>>(wb, nblocks, w16, xgrid, x, m, k, ldx, x16);
        chained = true;
    } else {
        x_to_f16_kernel<<<xgrid, 256, 0, ctx->stream>>>(x, m, k, ldx, x16);
        if (need_convert) {
            cq_status s2 = cq_is_k_format(qtype) ? launch_w_to_f16_k(ctx, qtype, w, n * (k / 256), w16) : launch_w_to_f16_more(ctx, qtype, order, w, n * (k / kQK), w16);
            if (s2 != CQ_OK) return s2;
        }
    }
    CQ_CUDA(ctx, cudaGetLastError());
    CUtensorMap tmA, tmB;
    const int bn = (m <= 64 && ctx->tune.gemm_variant != 1) ? 64 : 256;
    if (!make_map(&tmA, x16, m, k, BM) || !make_map(&tmB, w16, n, k, bn))
        return cq_fail(ctx, CQ_ERR_CUDA, "gemm: cuTensorMapEncodeTiled failed or is unavailable");
    static thread_local int configured_device = -1;
    if (configured_device != ctx->device) {
        CQ_CUDA(ctx, cudaFuncSetAttribute(gemm_f16_tn_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GemmCfg<256>::kSmem));
        CQ_CUDA(ctx, cudaFuncSetAttribute(gemm_f16_tn_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GemmCfg<64>::kSmem));
        configured_device = ctx->device;
    }
    dim3 grid((unsigned)((m + BM - 1) / BM), (unsigned)((n + bn - 1) / bn));
    if (bn == 256 && ctx->tune.gemm_variant == 0 && ctx->tune.gemm_pair) {
        // CTA pairs: 256 x 256 tiles, one per two SMs
        CUtensorMap tmBh;
        if (!make_map(&tmBh, w16, n, k, 128)) return cq_fail(ctx, CQ_ERR_CUDA, "gemm: cuTensorMapEncodeTiled failed or is unavailable");
        static thread_local int configured_pair = -1;
        static thread_local int max_clusters = 0;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr, cfg.numAttrs = 1;
        cfg.blockDim = dim3(GEMM_THREADS);
        cfg.dynamicSmemBytes = P2_SMEM;
        cfg.stream = ctx->stream;
        if (configured_pair != ctx->device) {
            CQ_CUDA(ctx, cudaFuncSetAttribute(gemm_f16_tn_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P2_SMEM));
            cfg.gridDim = dim3((unsigned)ctx->sm_count & ~1u);
            int nc = 0;
            CQ_CUDA(ctx, cudaOccupancyMaxActiveClusters(&nc, gemm_f16_tn_pair_kernel, &cfg));
            max_clusters = nc;
            configured_pair = ctx->device;
        }
        if (max_clusters > 0) {
            const int64_t ntiles = ((m + 255) / 256) * ((n + 255) / 256);
            const int64_t pairs = ntiles < max_clusters ? ntiles : max_clusters;
            cfg.gridDim = dim3((unsigned)(2 * pairs));
            if (chained && ctx->tune.pdl) cfg.numAttrs = 2;
            CQ_CUDA(ctx, cudaLaunchKernelEx(&cfg, gemm_f16_tn_pair_kernel, tmA, tmBh, y, (int)m, (int)n, (int)k, ldy, ctx->dev_err_devptr));
            return CQ_OK;
        }
    }
    if (bn == 256 && ctx->tune.gemm_variant != 2) {
        static thread_local int configured_p = -1;
        if (configured_p != ctx->device) {
            CQ_CUDA(ctx, cudaFuncSetAttribute(gemm_f16_tn_persistent_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GemmCfg<256>::kSmem));
            configured_p = ctx->device;
        }
        const int64_t ntiles = (int64_t)grid.x * grid.y;
        const unsigned ctas = (unsigned)(ntiles < ctx->sm_count ? ntiles : ctx->sm_count);
        gemm_f16_tn_persistent_kernel<<<ctas, GEMM_THREADS, GemmCfg<256>::kSmem, ctx->stream>>>(tmA, tmB, y, (int)m, (int)n, (int)k, ldy,
                                                                                               ctx->dev_err_devptr);
    } else if (bn == 64)
        gemm_f16_tn_kernel<64><<<grid, GEMM_THREADS, GemmCfg<64>::kSmem, ctx->stream>>>(tmA, tmB, y, (int)m, (int)n, (int)k, ldy, ctx->dev_err_devptr);
    else
        gemm_f16_tn_kernel<256><<<grid, GEMM_THREADS, GemmCfg<256>::kSmem, ctx->stream>>>(tmA, tmB, y, (int)m, (int)n, (int)k, ldy, ctx->dev_err_devptr);
    CQ_CUDA(ctx, cudaGetLastError());
    return CQ_OK;
}
