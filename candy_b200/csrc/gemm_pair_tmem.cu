// Batched quantized GEMM on CTA pairs, raw weight blocks dequantized into tensor memory:
// Y[m,n] = X[m,k] . W[n,k]^T for Q4_0 / Q8_0 weights, in one of two arithmetics (template parameter SPLIT):
//
//   SPLIT = false  CQ_ACT_F16: activations and weights rounded once to f16, f32 accumulation.
//   SPLIT = true   CQ_ACT_F32: both operands as the sum of two f16 numbers.  A weight d * q is a multiple of 2^-24 with
//                  at most 19 significant bits, so hi = f16(d q), lo = d q - hi hold it EXACTLY (lo is one fused
//                  multiply-add away from hi); an activation, scaled by a power of two per row so that the row's largest
//                  value sits just below 2^15, keeps 22 bits.  y = Xhi Whi + (Xlo Whi + Xhi Wlo); the dropped Xlo Wlo is
//                  2^-22 of the product.  The bracket has an accumulator of its own: the tensor core truncates when it
//                  adds, and small terms added to a large sum would each cost a truncation.
//
// Truncations go in one direction, two to a step of K = 16, so they add up with the length of the sum: for operands of one sign
// to 4.6e-9 of the result per value of k (512 rows, k = 28672: 6.2e-5; f32 additions of 32-term dots stay below 1e-6 there).  A
// tile's k range is therefore worked off in legs of at most 4096 values, which the epilogue adds up in f32; a tile of k = 4096 is
// one leg.  Against f64 (2-norm) at any k: operands of one sign at most 1.8e-5, centred ones 6e-7 .. 4e-6, where 15-bit block
// fixed point, which served these calls before, shows 4.1e-5.  512 x 4096 x 14336, us: whole sums 120, legs of 4096 127, of 2048
// (half the error) 140, of 1024 168, in one build; with the row scales out of the epilogue's way 119 for legs of 4096.
// CQ_ACT_F16 sums stay whole: two accumulators share them, and its operands' rounding, 2.9e-4, is what its results show.
//
// What bounds it: the tensor pipe for large batches (three products per term in SPLIT), the weight stream for small ones.
// The integer kernel that served CQ_ACT_F32 batches before has to scale every 32-term dot on the CUDA cores and stood at
// 120 TFLOP/s whatever the batch.
//
// A pair of CTAs (the two SMs of a TPC) works on 256 weight rows x NB batch rows, tcgen05.mma cta_group::2, M = 256:
//   each CTA   dequantizes ITS 128 weight rows into its own tensor memory (A operand) and loads HALF of the batch rows'
//              slab into its shared memory (B operand): the slab crosses L2 once per pair
//   warp 0     TMA, X slabs of 128 k (completion counted on the leader's barrier)
//   warp 1     TMA, raw blocks: [128 rows x 144 / 272 B] per 256 k
//   warps 2,3  of the leader: MMA issue.  The whole warp runs the loop and one lane issues: a loop that a lane runs alone starts
//              an MMA only every ~100-150 cycles, the pipe wants one every 64 (512 rows x 11008 x 4096, SPLIT: 125 -> 109 us).
//              SPLIT: one warp issues Xhi Whi, the other the two corrections; else they take alternate K = 16 steps.  Each
//              has its own accumulator.
//   DQ warps   groups of four (128 rows); group g owns A buffer g and converts every G-th stage of 128 k, so a group
//              converts while the tensor core works on the other buffers
//   8 warps    epilogue: lane = weight row, so a batch row's outputs leave in 128-byte runs
// Work is the list of (tile, 256-wide chunk of k), tile-major with the batch tiles of a weight group side by side, cut
// into equal contiguous shares per pair; partial tiles go to scratch and a small kernel adds them in pair order (the same
// bits from run to run).  Every wait is bounded.  Every barrier is waited on by the same threads for each of its phases.
//
// SPLIT and huge scales: f16 holds 65504.  A thread that meets a scale whose products could pass that (or inf / NaN) marks
// its weight row for the piece of work at hand, and the epilogue computes marked rows of it from the blocks in plain f32.
#include "gemm_raw.cuh"

namespace {

constexpr int GP_TILE = 256;    // weight rows per pair
constexpr int GP_EPW = 8;       // epilogue warps
constexpr int GP_LEG = 16;      // SPLIT: chunks that the tensor core adds up before an f32 addition does (see above)

template <int QT, bool SPLIT, int NB>
struct GpCfg {
    static constexpr int kBlockBytes = QT == CQ_Q4_0 ? kQ4Bytes : kQ8Bytes;
    static constexpr int kRowChunk = 8 * kBlockBytes;          // 144 / 272 bytes
    static constexpr int kWBytes = GP_ROWS * kRowChunk;
    static constexpr int kHalfWords = kRowChunk / 8;           // 32-bit words of four blocks
    static constexpr int kGroups = SPLIT ? 2 : 4;              // dequantizing groups = A buffers
    static constexpr int kACols = SPLIT ? 128 : 64;            // tensor-memory columns of an A buffer: hi (and lo)
    static constexpr int kWStages = QT == CQ_Q4_0 ? 4 : 2;     // even: without SPLIT the groups of a stage alternate with the chunk
    static constexpr int kBoxBytes = (NB / 2) * 128;           // 64 k of this CTA's batch rows
    static constexpr int kXBytes = (SPLIT ? 4 : 2) * kBoxBytes;
    static constexpr int kXStages = SPLIT ? 4 : 6;
    static constexpr int kWarpDq0 = 4, kWarpEp0 = kWarpDq0 + 4 * kGroups;
    static constexpr int kThreads = 32 * (kWarpEp0 + GP_EPW);
    static constexpr int kBars = 2 * kWStages + 2 * kXStages + 4 * kGroups + 2;
    static constexpr size_t kSmem = (size_t)kWStages * kWBytes + (size_t)kXStages * kXBytes + 1024 + 8 * kBars + 16 + 4 * GP_ROWS;
    static constexpr int kACol0 = 256;                         // accumulators: two of NB columns at 0
    static_assert(kSmem <= 232448 && 2 * NB <= kACol0 && kACol0 + kGroups * kACols <= 512, "shared / tensor memory");
};

// ---- activation pre-passes ---------------------------------------------------------------------------------
// Two 16-byte loads per eight values (value by value through a table of positions in constant memory: 128 rows x 4096 x 4096
// 16.9 us a call instead of 16.2, CQ_ACT_F32 128 x 4096 x 11008 48.7 instead of 45.7).
__global__ void __launch_bounds__(256) gp_x_f16_kernel(const float *__restrict__ x, int64_t m, int64_t k, int64_t ldx, int order,
                                                     __half *__restrict__ out) {
    pdl_launch_dependents();
    pdl_wait_prior();
    const int64_t per_row = k / 8, total = m * per_row;
    const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0 && ldx % 4 == 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t row = i / per_row, o8 = i - row * per_row;
        float v[8];
        load_permuted8(x + row * ldx + (o8 >> 2) * 32, (int)(o8 & 3), order, vec, v);
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const __half2 h = __floats2half2_rn(v[2 * j], v[2 * j + 1]);
            w[j] = *reinterpret_cast<const uint32_t *>(&h);
        }
        *reinterpret_cast<uint4 *>(out + row * k + o8 * 8) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// One CTA per row: largest magnitude, then x 2^e = hi + lo with 2^14 <= amax 2^e < 2^15 (e = 0 for a row of zeros or one
// that holds an infinity; infinities and NaNs make the row's results NaN).
// lo ends at f16's last bit, 2^-24: a value keeps 22 bits down to 2^-2 or so, and 2^-25 of absolute error below.  A 32-block
// whose largest value is under 2^-10 (2^-25 of the row's) would keep fewer than the 15 bits that it has in batches of up to
// eight rows (block fixed point).  Such a row's scale is handed over negative, and the epilogue computes the row in plain f32.
__global__ void __launch_bounds__(256) gp_x_split_kernel(const float *__restrict__ x, int64_t k, int64_t ldx, int order, __half *__restrict__ hi,
                                                       __half *__restrict__ lo, float *__restrict__ scale) {
    pdl_launch_dependents();
    pdl_wait_prior();
    __shared__ float red[8];
    const int64_t row = blockIdx.x;
    const float *src = x + row * ldx;
    const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0 && ldx % 4 == 0;
    float amax = 0.0f;
    if (vec) {
        for (int64_t i = threadIdx.x; i < k / 4; i += 256) {
            const float4 t = reinterpret_cast<const float4 *>(src)[i];
            amax = fmaxf(amax, fmaxf(fmaxf(fabsf(t.x), fabsf(t.y)), fmaxf(fabsf(t.z), fabsf(t.w))));
        }
    } else {
        for (int64_t i = threadIdx.x; i < k; i += 256) amax = fmaxf(amax, fabsf(src[i]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
    __syncthreads();
    amax = red[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) amax = fmaxf(amax, red[i]);
    int e = 0;
    if (amax > 0.0f && amax < INFINITY) e = min(14 - ilogbf(amax), 126);
    const float up = __int_as_float((127 + e) << 23);  // e in [-113, 126]
    bool low = false;
#pragma unroll 4
    for (int64_t o8 = threadIdx.x; o8 < k / 8; o8 += 256) {
        float v[8];
        load_permuted8(src + (o8 >> 2) * 32, (int)(o8 & 3), order, vec, v);
        uint32_t wh[4], wl[4];
        float top = 0.0f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float a = v[2 * j] * up, b = v[2 * j + 1] * up;
            top = fmaxf(top, fmaxf(fabsf(a), fabsf(b)));
            const __half2 h = __floats2half2_rn(a, b);
            const __half2 l = __floats2half2_rn(a - __low2float(h), b - __high2float(h));
            wh[j] = *reinterpret_cast<const uint32_t *>(&h);
            wl[j] = *reinterpret_cast<const uint32_t *>(&l);
        }
        *reinterpret_cast<uint4 *>(hi + row * k + o8 * 8) = make_uint4(wh[0], wh[1], wh[2], wh[3]);
        *reinterpret_cast<uint4 *>(lo + row * k + o8 * 8) = make_uint4(wl[0], wl[1], wl[2], wl[3]);
        // a block's 32 values lie in four neighbouring lanes (k is a multiple of 256: warps are in the loop as a whole)
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
        low |= top > 0.0f && top < 0x1p-10f;
    }
    low = __syncthreads_or(low && amax < INFINITY);
    if (threadIdx.x == 0) scale[row] = (low ? -1.0f : 1.0f) * __int_as_float((127 - e) << 23);
}

// q (an f16 pair of whole numbers) times the scale: the rounded product, and what the rounding took off (exact)
template <bool SPLIT>
__device__ __forceinline__ void gp_scale(__half2 q, __half2 d2, uint32_t &hi, uint32_t &lo) {
    const __half2 h = __hmul2(q, d2);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    if (SPLIT) {
        const __half2 l = __hfma2(q, d2, __hneg2(h));
        lo = *reinterpret_cast<const uint32_t *>(&l);
    }
}
template <bool SPLIT>
__device__ __forceinline__ void gp_dequant_q4(uint32_t n, __half2 d2, uint32_t *hi, uint32_t *lo) {
    __half2 q[4];
    gp_numbers_q4(n, q);
#pragma unroll
    for (int j = 0; j < 4; ++j) gp_scale<SPLIT>(q[j], d2, hi[j], lo[j]);
}
template <bool SPLIT>
__device__ __forceinline__ void gp_dequant_q8(uint32_t n, __half2 d2, uint32_t *hi, uint32_t *lo) {
    __half2 q[2];
    gp_numbers_q8(n, q);
#pragma unroll
    for (int j = 0; j < 2; ++j) gp_scale<SPLIT>(q[j], d2, hi[j], lo[j]);
}

__device__ __forceinline__ void tc_mma_f16_ts_pair(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
        "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// TMA load into THIS CTA's shared memory whose completion bytes are counted on a barrier of either CTA of the pair
__device__ __forceinline__ void tma_load_4d_pair(uint32_t smem_dst, const CUtensorMap *map, int x, int y, int z, int u, uint32_t bar_cluster_addr) {
    asm volatile(
        "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_dst),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(u), "r"(bar_cluster_addr)
        : "memory");
}

// A dot product over blocks [b0, b1) in plain f32, for marked weight rows and for batch rows of very different blocks.
template <int QT>
__device__ __noinline__ float gp_plain_dot(const uint8_t *wrow, const float *xrow, int order, int b0, int b1) {
    constexpr int BB = QT == CQ_Q4_0 ? kQ4Bytes : kQ8Bytes;
    float acc = 0.0f;
    for (int b = b0; b < b1; ++b) {
        const unsigned short *blk = reinterpret_cast<const unsigned short *>(wrow + (int64_t)b * BB);
        const float d = __half2float(__ushort_as_half(blk[0])), *xb = xrow + (int64_t)b * kQK;  // x: 16-byte aligned rows
#pragma unroll
        for (int j = 0; j < (BB - 2) / 2; ++j) {
            const int two = blk[1 + j];
            if (QT == CQ_Q4_0) {
                const bool inter = order == CQ_ORDER_GO_INTERLEAVED;  // bytes 2j, 2j + 1: values 4j .. 4j + 3, or 2j, 2j + 1 and 16 further
                const float2 u = *reinterpret_cast<const float2 *>(xb + (inter ? 4 * j : 2 * j)), v = *reinterpret_cast<const float2 *>(xb + (inter ? 4 * j + 2 : 2 * j + 16));
                const float n0 = d * (float)((two & 15) - 8), n1 = d * (float)(((two >> 4) & 15) - 8), n2 = d * (float)(((two >> 8) & 15) - 8),
                            n3 = d * (float)((two >> 12) - 8);
                acc = fmaf(n0, u.x, fmaf(inter ? n1 : n2, u.y, fmaf(inter ? n2 : n1, v.x, fmaf(n3, v.y, acc))));
            } else {
                const float2 u = *reinterpret_cast<const float2 *>(xb + 2 * j);
                acc = fmaf(d * (float)(signed char)(two & 0xFF), u.x, fmaf(d * (float)(signed char)(two >> 8), u.y, acc));
            }
        }
    }
    return acc;
}

template <int QT, bool SPLIT, int NB>
__global__ void __launch_bounds__(GpCfg<QT, SPLIT, NB>::kThreads, 1)
    gemm_pair_tmem_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const GpParams p) {
    using Cfg = GpCfg<QT, SPLIT, NB>;
    constexpr int WST = Cfg::kWStages, XST = Cfg::kXStages, G = Cfg::kGroups, HW = Cfg::kHalfWords, ROWCHUNK = Cfg::kRowChunk;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *smem_x = smem;                                          // XST slabs (1024-byte aligned boxes)
    uint8_t *smem_w = smem + (size_t)XST * Cfg::kXBytes;             // WST raw stages
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem_w + (size_t)WST * Cfg::kWBytes);
    uint64_t *w_full = bars, *w_empty = w_full + WST, *x_full = w_empty + WST, *x_empty = x_full + XST, *a_full = x_empty + XST,
             *a_empty = a_full + 2 * G, *d_full = a_empty + 2 * G, *d_empty = d_full + 1;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(d_empty + 1);
    // SPLIT: rows that the epilogue computes itself, [parity of the piece of work][epilogue warps of each half][row]
    volatile uint8_t *marked = reinterpret_cast<volatile uint8_t *>(tmem_slot + 4);

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const int pair = blockIdx.x >> 1;
    const int g0 = pair * p.per_share, g1 = min(g0 + p.per_share, p.total);
    const int nst = 2 * (g1 - g0);  // A / X stages of this share

    if (threadIdx.x == 0) {
        for (int s = 0; s < WST; ++s) {
            mbar_init(smem_u32(&w_full[s]), 1);
            mbar_init(smem_u32(&w_empty[s]), 8);      // the two groups that read a stage
        }
        for (int s = 0; s < XST; ++s) {
            mbar_init(smem_u32(&x_full[s]), 1);       // (used in the leader) its expect_tx; the bytes of both CTAs
            mbar_init(smem_u32(&x_empty[s]), 2);      // both issuers
        }
        for (int b = 0; b < 2 * G; ++b) {             // per A buffer: one for each half of its 128 k
            mbar_init(smem_u32(&a_full[b]), 8);       // (leader) the group's four warps in both CTAs
            mbar_init(smem_u32(&a_empty[b]), 2);
        }
        mbar_init(smem_u32(d_full), 2);
        mbar_init(smem_u32(d_empty), 2 * GP_EPW);     // (leader) the epilogue warps of both CTAs
        fence_mbar_init();
        fence_proxy_async();
    }
    if (SPLIT && threadIdx.x < 4 * GP_ROWS) marked[threadIdx.x] = 0;
    __syncthreads();
    cluster_sync_all();  // the peer's barriers exist before anything of this CTA can signal them
    if (warp == 1) tmem_alloc_pair(smem_u32(tmem_slot), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents();  // not before the tensor memory is ours: a dependent may want some too

    // the piece of work that starts at item g: what is left of its tile in this share, SPLIT: in legs
    auto segment = [&](int g, int &tile, int &c0, int &cn) {
        tile = g / p.nchunks;
        c0 = g - tile * p.nchunks;
        cn = min(p.nchunks - c0, g1 - g);
        if (SPLIT && cn > GP_LEG) {
            const int legs = (cn + GP_LEG - 1) / GP_LEG;
            cn = (cn + legs - 1) / legs;
        }
    };

    if (warp == 0) {
        // ---- TMA, X: this CTA's half of the batch rows, 128 k per stage ----
        if (lane == 0) {
            pdl_wait_prior();
            bool ok = true;
            int i = 0;
            for (; i < nst; ++i) {
                const int g = g0 + (i >> 1), tile = g / p.nchunks, c = g - tile * p.nchunks;
                const int s = i % XST;
                if (i >= XST && !mbar_wait_bounded(smem_u32(&x_empty[s]), ((i / XST) - 1) & 1)) {
                    atomicExch(p.err, kDevErrEmptyWait);
                    ok = false;
                    break;
                }
                const uint32_t lead = mapa_shared(smem_u32(&x_full[s]), 0);
                if (rank == 0) mbar_expect_tx(smem_u32(&x_full[s]), 2 * Cfg::kXBytes);
                const uint32_t dst = smem_u32(smem_x + (size_t)s * Cfg::kXBytes);
                tma_load_4d_pair(dst, &tmX, 0, (tile % p.mtiles) * NB + (int)rank * (NB / 2), 4 * c + 2 * (i & 1), 0, lead);
            }
            if (rank == 0 && ok)  // the leader's barriers count the bytes of both CTAs: leave when the last ones have landed
                for (int j = i > XST ? i - XST : 0; j < i; ++j)
                    if (!mbar_wait_bounded(smem_u32(&x_full[j % XST]), (j / XST) & 1)) {
                        atomicExch(p.err, kDevErrDrain);
                        break;
                    }
        }
    } else if (warp == 1) {
        // ---- TMA, raw blocks of this CTA's 128 weight rows, 256 k per stage ----
        if (lane == 0) {
            bool ok = true;
            int i = 0;
            for (; i < nst / 2; ++i) {
                const int g = g0 + i, tile = g / p.nchunks, c = g - tile * p.nchunks;
                const int s = i % WST;
                if (i >= WST && !mbar_wait_bounded(smem_u32(&w_empty[s]), ((i / WST) - 1) & 1)) {
                    atomicExch(p.err, kDevErrEmptyWait);
                    ok = false;
                    break;
                }
                mbar_expect_tx(smem_u32(&w_full[s]), Cfg::kWBytes);
                // rows past n are outside the tensor: zero fill
                tma_load_2d(smem_u32(smem_w + (size_t)s * Cfg::kWBytes), &tmW, c * (ROWCHUNK / 2), (tile / p.mtiles) * GP_TILE + (int)rank * GP_ROWS,
                            smem_u32(&w_full[s]));
            }
            if (ok)
                for (int j = i > WST ? i - WST : 0; j < i; ++j)
                    if (!mbar_wait_bounded(smem_u32(&w_full[j % WST]), (j / WST) & 1)) {
                        atomicExch(p.err, kDevErrDrain);
                        break;
                    }
        }
    } else if (warp < Cfg::kWarpDq0) {
        // ---- MMA issue (leader only): the whole warp runs the loop, one lane issues ----
        if (rank == 0) {
            constexpr uint32_t idesc = idesc_f16(256, NB);
            const int e = warp - 2;
            const uint32_t acc = tmem_base + (uint32_t)(e * NB);
            int i = 0, seg = 0;
            bool ok = true;
            for (int g = g0; g < g1 && ok; ++seg) {
                int tile, c0, cn;
                segment(g, tile, c0, cn);
                g += cn;
                if (seg >= 1 && !__all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(d_empty), (seg - 1) & 1))) {  // the epilogue has read the accumulators
                    if (lane == 0) atomicExch(p.err, kDevErrMma);
                    break;
                }
                tc_fence_after();
                for (int c = 0; c < 2 * cn; ++c, ++i) {
                    const int s = i % XST, b = i % G;
                    const uint64_t xh = smem_desc_k128(smem_u32(smem_x + (size_t)s * Cfg::kXBytes));
                    const uint32_t ah = tmem_base + (uint32_t)(Cfg::kACol0 + b * Cfg::kACols);
                    // K = 16 step j of the stage: box j / 4 of the slab, 32-byte column j % 4
                    auto at = [&](int j) { return (uint64_t)((j >> 2) * (Cfg::kBoxBytes / 16) + (j & 3) * 2); };
#pragma unroll
                    for (int hh = 0; hh < 2; ++hh) {
                        const bool there = (hh || mbar_wait_bounded(smem_u32(&x_full[s]), (i / XST) & 1)) && mbar_wait_bounded(smem_u32(&a_full[2 * b + hh]), (i / G) & 1);
                        if (!__all_sync(0xffffffffu, there)) {
                            if (lane == 0) atomicExch(p.err, kDevErrFullWait);
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        if (elect_one()) {
                            if (SPLIT) {
                                if (e == 0) {
#pragma unroll
                                    for (int j = 4 * hh; j < 4 * hh + 4; ++j) tc_mma_f16_ts_pair(acc, ah + 8 * j, xh + at(j), idesc, (c | j) != 0);
                                } else {
                                    const uint64_t xl = xh + (uint64_t)(2 * Cfg::kBoxBytes / 16);
#pragma unroll
                                    for (int j = 4 * hh; j < 4 * hh + 4; ++j) {
                                        tc_mma_f16_ts_pair(acc, ah + 8 * j, xl + at(j), idesc, (c | j) != 0);
                                        tc_mma_f16_ts_pair(acc, ah + 64 + 8 * j, xh + at(j), idesc, 1);
                                    }
                                }
                            } else {
#pragma unroll
                                for (int j2 = 2 * hh; j2 < 2 * hh + 2; ++j2) {
                                    const int j = 2 * j2 + e;
                                    tc_mma_f16_ts_pair(acc, ah + 8 * j, xh + at(j), idesc, (c | j2) != 0);
                                }
                            }
                            tc_commit_pair(smem_u32(&a_empty[2 * b + hh]), 3);
                            if (hh == 1) {
                                tc_commit_pair(smem_u32(&x_empty[s]), 3);
                                if (c == 2 * cn - 1) tc_commit_pair(smem_u32(d_full), 3);
                            }
                        }
                        __syncwarp();
                    }
                    if (!ok) break;
                }
            }
        }
    } else if (warp < Cfg::kWarpEp0) {
        // ---- dequantize: thread = weight row, group = every G-th stage ----
        const int grp = (warp - Cfg::kWarpDq0) >> 2, quarter = warp & 3, r = quarter * 32 + lane;
        const uint32_t a_t = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(Cfg::kACol0 + grp * Cfg::kACols);
        const uint32_t lead_full = mapa_shared(smem_u32(&a_full[2 * grp]), 0);
        bool ok = true;
        for (int i = grp; i < nst && ok; i += G) {
            const int c = i >> 1, h = i & 1, s = c % WST;
            if (!mbar_wait_sleep(smem_u32(&w_full[s]), (c / WST) & 1, 20)) {
                if (lane == 0) atomicExch(p.err, kDevErrFullWait);
                break;
            }
            uint32_t w[HW];  // four blocks = 72 / 136 bytes, 8-byte aligned
            const uint32_t src = smem_u32(smem_w + (size_t)s * Cfg::kWBytes + r * ROWCHUNK + h * (ROWCHUNK / 2));
#pragma unroll
            for (int j = 0; j < HW / 2; ++j)
                asm volatile("ld.volatile.shared.v2.u32 {%0, %1}, [%2];" : "=r"(w[2 * j]), "=r"(w[2 * j + 1]) : "r"(src + 8 * j) : "memory");
            // The two halves of the buffer (two blocks, 64 k each) are handed over one by one: the tensor core works on the first
            // while the second is converted, and the next round begins when the first is free again.
            bool big = false;
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                if (i >= G && !mbar_wait_sleep(smem_u32(&a_empty[2 * grp + hh]), ((i / G) - 1) & 1, 20)) {
                    if (lane == 0) atomicExch(p.err, kDevErrMma);
                    ok = false;
                    break;
                }
                tc_fence_after();
#pragma unroll
                for (int blk = 2 * hh; blk < 2 * hh + 2; ++blk) {
                    // two blocks in 9 (Q4_0) / 17 (Q8_0) words: the first starts on a word, its values two bytes in; the second
                    // starts two bytes into the middle word, its values on the next one
                    constexpr int PW = HW / 2, VW = (PW - 1) / 2;
                    const uint32_t *wq = w + PW * hh;
                    const unsigned short db = (unsigned short)((blk & 1) ? (wq[VW] >> 16) : (wq[0] & 0xFFFFu));
                    const __half2 d2 = __half2half2(__ushort_as_half(db));
                    // products of |d| >= 8192 (Q4_0: 8 d) / 512 (Q8_0: 128 d) could pass f16's largest value; inf and NaN are larger still
                    if (SPLIT) big |= (db & 0x7FFFu) >= (QT == CQ_Q4_0 ? 0x7000u : 0x6000u);
                    uint32_t hi[16], lo[16];
#pragma unroll
                    for (int j = 0; j < VW; ++j) {
                        const uint32_t v = (blk & 1) ? wq[VW + 1 + j] : __funnelshift_r(wq[j], wq[j + 1], 16);
                        if (QT == CQ_Q4_0) gp_dequant_q4<SPLIT>(v, d2, hi + 4 * j, lo + 4 * j);
                        else gp_dequant_q8<SPLIT>(v, d2, hi + 2 * j, lo + 2 * j);
                    }
                    tmem_st16(a_t + (uint32_t)(16 * blk), hi);
                    if (SPLIT) tmem_st16(a_t + (uint32_t)(64 + 16 * blk), lo);
                }
                if (SPLIT && hh == 1 && big) {
                    // The mark is for this piece alone.  Its parity is enough: work on the piece after the next begins when the tensor
                    // core has used stages of the next one, which it starts on after the epilogue has read (and cleared) this one's.
                    int g = g0, odd = 0, tile, c0, cn;
                    for (segment(g, tile, c0, cn); g + cn <= g0 + c; segment(g, tile, c0, cn)) g += cn, odd ^= 1;
                    marked[2 * odd * GP_ROWS + r] = 1;
                    marked[(2 * odd + 1) * GP_ROWS + r] = 1;
                }
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive_cluster(lead_full + 8 * hh);
                    // The raw stage is free too: every word of it has gone through a finished store.  (Handing it back right after the
                    // loads would need an instruction that consumes all of them first: an arrive does not wait for loads in flight.)
                    if (hh == 1) mbar_arrive(smem_u32(&w_empty[s]));
                }
            }
        }
    } else {
        // ---- epilogue: lane = weight row, two warps per 32 rows take alternate pieces of 16 columns ----
        pdl_wait_prior();  // y and the partial tiles may still be read by earlier kernels; the row scales are the pre-pass's
        const int quarter = warp & 3, half = (warp - Cfg::kWarpEp0) >> 2, r = quarter * 32 + lane;
        const uint32_t lead_empty = mapa_shared(smem_u32(d_empty), 0);
        const int first_tile = g0 / p.nchunks;
        int seg = 0;
        for (int g = g0; g < g1; ++seg) {
            int tile, c0, cn;
            segment(g, tile, c0, cn);
            const bool more = SPLIT && g != g0 && c0 != 0;  // a further leg of a tile: added to what the same thread has stored
            g += cn;
            const int group = tile / p.mtiles, col0 = (tile - group * p.mtiles) * NB;
            const int row_in_tile = (int)rank * GP_ROWS + r, row = group * GP_TILE + row_in_tile;
            // whole k range in this share -> y, otherwise one of this pair's two partial slots
            const bool direct = tile * p.nchunks >= g0 && (tile + 1) * p.nchunks <= g1;
            const int64_t ld = direct ? p.ldy : GP_TILE;
            float *dst = direct ? p.y + (int64_t)col0 * p.ldy + row : p.part + (int64_t)(2 * pair + (tile == first_tile ? 0 : 1)) * NB * GP_TILE + row_in_tile;
            const float bias = direct && !more && p.bias && row < p.n ? p.bias[row] : 0.0f;
            auto column = [&](int i, int j) { return 16 * (half + 2 * i) + j; };  // of this warp's piece i
            // SPLIT takes all of its columns into registers before it stores any, so that the tensor core can go on, and fetches what
            // the legs before have stored while it waits for this one (with loads and stores between the pieces a leg's epilogue took
            // longer than the leg: 512 x 4096 x 14336 171 us instead of 119; at k = 4096, one leg, 512 x 11008 105 -> 92).
            // The row scales are fetched then too, two pieces of 16 to a warp's lanes, and handed round by shuffles.
            constexpr int HELD = SPLIT ? NB / 32 : 1;
            float v[HELD][16], scales[(HELD + 1) / 2];
            if constexpr (SPLIT) {
#pragma unroll
                for (int i = 0; i < (HELD + 1) / 2; ++i) scales[i] = p.xscale[min(col0 + column(2 * i + (HELD > 1 ? lane >> 4 : 0), lane & 15), p.m - 1)];
#pragma unroll
                for (int i = 0; i < HELD; ++i)
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[i][j] = more && row < p.n && col0 + column(i, j) < p.m ? dst[column(i, j) * ld] : bias;
            }
            if (!__all_sync(0xffffffffu, mbar_wait_sleep(smem_u32(d_full), seg & 1, 100))) {
                if (lane == 0) atomicExch(p.err, kDevErrMma);
                break;
            }
            tc_fence_after();
            const uint32_t lanes = tmem_base + ((uint32_t)(quarter * 32) << 16);
            if constexpr (SPLIT) {
                volatile uint8_t *mark = marked + (2 * (seg & 1) + half) * GP_ROWS + r;
                const bool mine = *mark != 0;
                if (mine) *mark = 0;
                bool low = scales[0] < 0.0f;
                if (HELD > 2) low |= scales[HELD > 2 ? 1 : 0] < 0.0f;
                low = __any_sync(0xffffffffu, low);
                const bool plain = mine || low;  // some results are computed below
#pragma unroll
                for (int e = 0; e < HELD * 16; e += 8) {
                    const int i = e >> 4, j0 = e & 15;
                    uint32_t a[8], b[8];
                    tmem_ld8_async(lanes + (uint32_t)column(i, j0), a);
                    tmem_ld8_async(lanes + (uint32_t)column(i, j0) + NB, b);
                    tmem_wait_ld();
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float sc = __shfl_sync(0xffffffffu, scales[i / 2], 16 * (i & 1) + j0 + j);
                        v[i][j0 + j] += mine || sc < 0.0f ? 0.0f : (__uint_as_float(a[j]) + __uint_as_float(b[j])) * sc;
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(lead_empty);
#pragma unroll
                for (int i = 0; i < HELD; ++i)
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (row < p.n && col0 + column(i, j) < p.m) dst[column(i, j) * ld] = v[i][j];
                if (plain && row < p.n) {
                    // marked rows, and batch rows that the tensor core does not take
                    for (int c = 0; c < NB / 2; ++c) {
                        const int cc = column(c >> 4, c & 15), xr = col0 + cc;
                        if (xr >= p.m || !(mine || p.xscale[xr] < 0.0f)) continue;
                        dst[cc * ld] += gp_plain_dot<QT>(p.w + (int64_t)row * (p.k / kQK) * Cfg::kBlockBytes, p.x + (int64_t)xr * p.ldx, p.order, c0 * 8,
                                                         (c0 + cn) * 8);
                    }
                }
                __syncwarp();
            } else {
#pragma unroll 1
                for (int c = half; c < NB / 16; c += 2) {
                    uint32_t v0[16], v1[16];
                    tmem_ld16_async(lanes + (uint32_t)(c * 16), v0);
                    tmem_ld16_async(lanes + (uint32_t)(c * 16) + NB, v1);
                    tmem_wait_ld();
                    if (c + 2 >= NB / 16) {  // this warp's last piece is in registers
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive_cluster(lead_empty);
                    }
                    if (row < p.n) {
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (col0 + c * 16 + j < p.m) dst[(int64_t)(c * 16 + j) * ld] = __uint_as_float(v0[j]) + __uint_as_float(v1[j]) + bias;
                    }
                    __syncwarp();
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();  // neither CTA leaves (or frees tensor memory) while the pair's MMAs may still use it
    if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
}

template <int QT, bool SPLIT, int NB>
cq_status gp_run(cq_ctx *ctx, const float *x, int64_t m, int64_t k, int64_t ldx, int order, const void *w, int64_t n, float *y, int64_t ldy) {
    using Cfg = GpCfg<QT, SPLIT, NB>;
    auto kern = gemm_pair_tmem_kernel<QT, SPLIT, NB>;
    static thread_local int configured = -1, max_pairs = 0;
    if (configured != ctx->device) {
        CQ_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::kSmem));
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2, attr[0].val.clusterDim.y = 1, attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr, cfg.numAttrs = 1;
        cfg.gridDim = dim3((unsigned)ctx->sm_count & ~1u), cfg.blockDim = dim3(Cfg::kThreads), cfg.dynamicSmemBytes = Cfg::kSmem;
        int nc = 0;
        CQ_CUDA(ctx, cudaOccupancyMaxActiveClusters(&nc, kern, &cfg));
        if (nc < 1) return cq_fail(ctx, CQ_ERR_CUDA, "gemm: no CTA pair fits this device");
        max_pairs = nc;
        configured = ctx->device;
    }
    GpParams p = {};
    p.y = y, p.ldy = ldy, p.x = x, p.w = static_cast<const uint8_t *>(w), p.ldx = ldx;
    p.m = (int)m, p.n = (int)n, p.k = (int)k, p.order = order, p.err = ctx->dev_err_devptr, p.bias = ctx->bias;
    const size_t x_bytes = (((size_t)m * k * 2) + 1023) & ~size_t(1023);
    const size_t scale_bytes = SPLIT ? (((size_t)m * 4) + 1023) & ~size_t(1023) : 0;
    const size_t operand_bytes = (SPLIT ? 2 : 1) * x_bytes + scale_bytes;
    GpShares sh;
    cq_status s = gp_share_out(ctx, p, GP_TILE, NB, max_pairs, operand_bytes, sh);
    if (s == CQ_OK) s = cq_reserve_scratch(ctx, operand_bytes + sh.part_bytes);
    if (s != CQ_OK) return s;
    uint8_t *base = static_cast<uint8_t *>(ctx->scratch);
    __half *xh = reinterpret_cast<__half *>(base), *xl = reinterpret_cast<__half *>(base + (SPLIT ? x_bytes : 0));
    float *scale = reinterpret_cast<float *>(base + (SPLIT ? 2 : 1) * x_bytes);
    p.part = reinterpret_cast<float *>(reinterpret_cast<uint8_t *>(scale) + scale_bytes);
    p.xscale = scale;
    CUtensorMap tmW, tmX;
    if (!gp_w_map(&tmW, w, n, (k / kQK) * Cfg::kBlockBytes, Cfg::kRowChunk) || !gp_x_map(&tmX, xh, m, k, SPLIT ? x_bytes : 0, NB / 2, 2))
        return cq_fail(ctx, CQ_ERR_CUDA, "gemm: cuTensorMapEncodeTiled failed or is unavailable");
    const int ord = QT == CQ_Q4_0 ? order : 2;
    if (SPLIT) {
        s = gp_launch(ctx, gp_x_split_kernel, dim3((unsigned)m), 256, 0, false, x, k, ldx, ord, xh, xl, scale);
    } else {
        const int64_t items = m * (k / 8), cap = (int64_t)ctx->sm_count * 8;
        s = gp_launch(ctx, gp_x_f16_kernel, dim3((unsigned)((items + 255) / 256 < cap ? (items + 255) / 256 : cap)), 256, 0, false, x, m, k, ldx, ord, xh);
    }
    if (s != CQ_OK) return s;
    s = gp_launch(ctx, kern, dim3(2 * sh.shares), Cfg::kThreads, Cfg::kSmem, true, tmW, tmX, p);
    if (s == CQ_OK && sh.cut) s = gp_launch(ctx, gp_sum_kernel<GP_TILE, NB>, dim3((unsigned)sh.tiles, NB / 4), 256, 0, false, p);
    if (s == CQ_OK && p.bias) ctx->bias_done = true;
    return s;
}

}  // namespace

bool gemm_pair_tmem_supported(int qtype, int64_t k, const void *w) {
    // row starts on 16 bytes (the tensor map's strides) and whole chunks of 256 values
    return (qtype == CQ_Q4_0 || qtype == CQ_Q8_0) && k % GP_CHUNK == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0;
}

cq_status launch_gemm_pair_tmem(cq_ctx *ctx, int qtype, int order, bool split, const float *x, int64_t m, int64_t k, int64_t ldx, const void *w, int64_t n,
                                float *y, int64_t ldy) {
    if ((reinterpret_cast<uintptr_t>(x) & 3) != 0 || (reinterpret_cast<uintptr_t>(y) & 3) != 0)
        return cq_fail(ctx, CQ_ERR_INVALID_ARG, "gemm: misaligned pointer");
#define CQ_GP(QT, SP)                                                                                \
    return m <= 32   ? gp_run<QT, SP, 32>(ctx, x, m, k, ldx, order, w, n, y, ldy)                    \
           : m <= 64 ? gp_run<QT, SP, 64>(ctx, x, m, k, ldx, order, w, n, y, ldy)                    \
                     : gp_run<QT, SP, 128>(ctx, x, m, k, ldx, order, w, n, y, ldy)
    if (qtype == CQ_Q4_0) {
        if (split) CQ_GP(CQ_Q4_0, true);
        CQ_GP(CQ_Q4_0, false);
    }
    if (split) CQ_GP(CQ_Q8_0, true);
    CQ_GP(CQ_Q8_0, false);
#undef CQ_GP
}
