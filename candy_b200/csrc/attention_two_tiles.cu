// Prefill attention with two tiles of 128 query rows per CTA, the same contract as attention_prefill.cu (which serves small
// problems, V tiles that the tensor maps cannot address, and long rows of keys).
//
// One tile alone leaves the tensor core idle during its softmax and the other way round.  Here two tiles of the same head take
// turns, and each K and V tile is fetched once for both:
//   warp 0      TMA: the two Q tiles, K tiles into a three-stage ring, V tiles into a two-stage ring
//   warp 1      tcgen05.mma issue, tile by tile: O += P V(j), then S = Q K(j+1)^T into the columns that P has left (MMAs of one
//               thread execute in order); the whole warp runs the loop and one lane issues
//   warps 4-11  softmax of tile 0, warps 12-19 of tile 1: thread = (query row, half of the scores of a key tile).  p = ex2 of
//               the scaled difference goes back as 16-bit pairs over the first half of the scores' own tensor-memory columns
// p is taken relative to the row's maximum so far, the row's largest p is exactly 1, and the accumulators are rescaled wherever a
// key tile raises a maximum, by the softmax threads before they hand their p over: an output as near to 64 bits as one tile's.
// (With a reference that moves only when p would pass 2^13 the scores' maxima and the rescaling are saved, 453 us for 517 in the
// first shape below, but the largest p is rounded too: 2.05e-3 -> 2.09e-3 of the result in bf16, 2.56e-4 -> 2.61e-4 in f16.)
// The output accumulates in tensor memory over all key tiles, where the tensor core truncates as it adds: 6e-9 of the sum per key
// for values of one sign, 1e-9 for mixed ones.  Rows of up to 2048 keys (f16) / 8192 (bf16) come here, where that adds at most
// 0.3 % to the error that the rounding of p and of the result leaves (positive values, f16, 4096 keys: 1.767e-4 -> 1.784e-4, four
// times as much as at 2048; mixed ones 2.855e-4 either way).
//
// us, one tile per CTA -> two, sustained (in bursts): 2 x 64/8 heads x 4096 causal bf16 645 -> 557 (616 -> 517); 32 heads x 2048 causal
// f16 47 -> 39; 32/8 heads x 4096 of 64 causal bf16 141 -> 103.  What was tried (us, first shape, bursts): every p on the
// special-function unit 516, a half / a third / a quarter / a fifth on the f32 pipes 550 / 517 / 518 / 522 (32 x 2048: 46.5, 48, 45,
// 45.5, 46).
// Persistent CTAs, items (256 query rows, head, batch) heavy first and in alternating directions, as in attention_prefill.cu:
// rings, phases and tensor memory carry on from item to item.  Every wait is bounded; tensor memory is always freed.
#include "attention.cuh"

namespace {

constexpr int F2_THREADS = 640;
constexpr int F2_KS = 3, F2_VS = 2;
// registers per thread: launched with 96; the softmax warps take from the four control warps
constexpr int F2_REGS_LAUNCH = 96, F2_REGS_CONTROL = 64, F2_REGS_SOFTMAX = 104;
static_assert(128 * F2_REGS_CONTROL + 512 * F2_REGS_SOFTMAX <= F2_THREADS * F2_REGS_LAUNCH, "registers of the block");
constexpr int F2_TMA = 0, F2_MMA = 1, F2_SOFTMAX = 4;  // warps

template <int D>
struct F2Cfg {
    static constexpr int kSlabs = D / 64;                 // 64-wide slabs of the head dimension
    static constexpr int kTile = kSlabs * 128 * 128;      // bytes of a Q, K or V tile
    static constexpr size_t kSmem = (size_t)(2 + F2_KS + F2_VS) * kTile + 256 /* barriers */ + 2 * 2 * FA_M * 4 /* half rows */;
    static constexpr uint32_t kColS = 0, kColO = 256;     // 128 columns of scores (and p) a tile, D of output
    static_assert(kSmem <= 232448 && kColO + 2 * D <= 512, "shared / tensor memory");
};

__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t *r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
        "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
        "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}

__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// 2^x of two numbers on the f32 pipes: x = whole + f with |f| <= 1/2 by adding and taking off 1.5 * 2^23, 2^f by a polynomial
// (Remez exchange for the relative error on [-1/2, 1/2]: 7.5e-8, in f32 arithmetic 2.1e-7, as ex2.approx), the whole number
// as the exponent of a factor.  Below -127 the factor is 0; NaN stays NaN.  For x < 128: here no x is above a rounding of 0.
__device__ __forceinline__ uint64_t ex2_poly2(uint64_t x) {
    float a, b;
    unpack2(x, a, b);
    asm("max.NaN.f32 %0, %0, %1;" : "+f"(a) : "f"(-127.0f));
    asm("max.NaN.f32 %0, %0, %1;" : "+f"(b) : "f"(-127.0f));
    x = pack2(a, b);
    const uint64_t t = add2(x, dup2(12582912.0f)), f = fma2(add2(t, dup2(-12582912.0f)), dup2(-1.0f), x);
    uint64_t y = fma2(f, dup2(0x1.5c08e6p-10f), dup2(0x1.3d0c52p-7f));
    y = fma2(y, f, dup2(0x1.c6b6e4p-5f));
    y = fma2(y, f, dup2(0x1.ebf918p-3f));
    y = fma2(y, f, dup2(0x1.62e428p-1f));
    y = fma2(y, f, dup2(0x1.000002p+0f));
    unpack2(t, a, b);
    return mul2(y, pack2(__int_as_float((__float_as_int(a) << 23) + 0x3F800000), __int_as_float((__float_as_int(b) << 23) + 0x3F800000)));
}

template <int D, bool BF16>
__global__ void __launch_bounds__(F2_THREADS, 1)
    fmha_two_tiles_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const FaParams p) {
    using Cfg = F2Cfg<D>;
    constexpr int SLABS = Cfg::kSlabs;
    extern __shared__ __align__(1024) uint8_t smem[];  // (no room to align it by hand)
    if (smem_u32(smem) & 1023) {
        if (threadIdx.x == 0) atomicExch(p.err, kDevErrMma);
        return;
    }
    uint8_t *sm_q = smem;                                   // [2]
    uint8_t *sm_k = sm_q + 2 * Cfg::kTile;                  // [F2_KS]
    uint8_t *sm_v = sm_k + (size_t)F2_KS * Cfg::kTile;      // [F2_VS]
    float *sm_half = reinterpret_cast<float *>(sm_v + (size_t)F2_VS * Cfg::kTile);  // [2 tiles][2 halves][128]: maxima or sums of half rows
    uint64_t *bars = reinterpret_cast<uint64_t *>(sm_half + 4 * FA_M);
    uint64_t *q_full = bars, *q_empty = q_full + 2, *k_full = q_empty + 2, *k_empty = k_full + F2_KS, *v_full = k_empty + F2_KS, *v_empty = v_full + F2_VS,
             *s_full = v_empty + F2_VS, *p_full = s_full + 2, *o_done = p_full + 2, *o_free = o_done + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(o_free + 2);

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int off = p.seqlen_k - p.seqlen_q;  // causal: key j is visible to row i iff j <= i + off
    const int nq = (p.seqlen_q + 2 * FA_M - 1) / (2 * FA_M), hb = p.h * p.b, items = nq * hb;
    // item -> its first query row, head, batch and the key tiles of its two query tiles
    auto item_at = [&](int w, int &q0, int &head, int &batch, int (&nt)[2]) {
        const int qt = nq - 1 - w / hb, rem = w % hb;
        head = rem % p.h, batch = rem / p.h;
        q0 = qt * 2 * FA_M;
        const int all = (p.seqlen_k + FA_N - 1) / FA_N;
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            nt[x] = all;
            if (p.causal) {
                const int lim = q0 + (x + 1) * FA_M + off;  // keys >= lim are masked for every row of this tile
                nt[x] = min(all, lim <= 0 ? 0 : (lim + FA_N - 1) / FA_N);
            }
            if (q0 + x * FA_M >= p.seqlen_q) nt[x] = 0;
        }
    };
    const int kv_group = p.h / p.h_k;
    auto item_of_round = [&](int rd) { return (rd & 1) ? (rd + 1) * (int)gridDim.x - 1 - (int)blockIdx.x : rd * (int)gridDim.x + (int)blockIdx.x; };

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int x = 0; x < 2; ++x) {
            mbar_init(smem_u32(&q_full[x]), 1);
            mbar_init(smem_u32(&q_empty[x]), 1);
            mbar_init(smem_u32(&s_full[x]), 1);
            mbar_init(smem_u32(&p_full[x]), 8);
            mbar_init(smem_u32(&o_done[x]), 1);
            mbar_init(smem_u32(&o_free[x]), 8);
        }
        for (int s = 0; s < F2_KS; ++s) {
            mbar_init(smem_u32(&k_full[s]), 1);
            mbar_init(smem_u32(&k_empty[s]), 1);
        }
        for (int s = 0; s < F2_VS; ++s) {
            mbar_init(smem_u32(&v_full[s]), 1);
            mbar_init(smem_u32(&v_empty[s]), 1);
        }
        fence_mbar_init();
        fence_proxy_async();
    }
    if (warp == F2_MMA) tmem_alloc(smem_u32(tmem_slot), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp < F2_SOFTMAX) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(F2_REGS_CONTROL));
        if (warp == F2_TMA) {
            if (lane == 0) {
                pdl_wait_prior();  // Q, K and V come from earlier kernels
                bool ok = true;
                int g = 0, qi[2] = {0, 0};  // key tiles, and items of either query tile, loaded so far
                for (int rd = 0; rd * (int)gridDim.x < items && ok; ++rd) {
                    const int w = item_of_round(rd);
                    if (w >= items) continue;
                    int q0, head, batch, nt[2];
                    item_at(w, q0, head, batch, nt);
                    const int n = max(nt[0], nt[1]), kv_head = head / kv_group;
                    if (n == 0) continue;
                    auto load_q = [&](int x) {
                        if (nt[x] == 0 || !ok) return;
                        if (qi[x] >= 1 && !mbar_wait_sleep(smem_u32(&q_empty[x]), (qi[x] - 1) & 1, 100)) {
                            atomicExch(p.err, kDevErrEmptyWait);
                            ok = false;
                            return;
                        }
                        mbar_expect_tx(smem_u32(&q_full[x]), Cfg::kTile);
#pragma unroll
                        for (int c = 0; c < SLABS; ++c)
                            tma_load_4d(smem_u32(sm_q + x * Cfg::kTile + c * (FA_M * 128)), &tmQ, c * 64, head, q0 + x * FA_M, batch, smem_u32(&q_full[x]));
                        ++qi[x];
                    };
                    auto load = [&](int t, const CUtensorMap &map, uint8_t *ring, uint64_t *full, uint64_t *empty, int stages) {
                        if (!ok) return;
                        const int gt = g + t, s = gt % stages;
                        if (gt >= stages && !mbar_wait_sleep(smem_u32(&empty[s]), ((gt / stages) - 1) & 1, 100)) {
                            atomicExch(p.err, kDevErrEmptyWait);
                            ok = false;
                            return;
                        }
                        mbar_expect_tx(smem_u32(&full[s]), Cfg::kTile);
#pragma unroll
                        for (int c = 0; c < SLABS; ++c)
                            tma_load_4d(smem_u32(ring + (size_t)s * Cfg::kTile + c * (FA_N * 128)), &map, c * 64, kv_head, t * FA_N, batch, smem_u32(&full[s]));
                    };
                    load_q(0);
                    load(0, tmK, sm_k, k_full, k_empty, F2_KS);
                    load_q(1);
                    for (int t = 0; t < n && ok; ++t) {
                        if (t + 1 < n) load(t + 1, tmK, sm_k, k_full, k_empty, F2_KS);
                        load(t, tmV, sm_v, v_full, v_empty, F2_VS);
                    }
                    g += n;
                }
                // leave only when nothing is in flight into this CTA's shared memory
                bool landed = ok;
                for (int x = 0; x < 2; ++x)
                    if (landed && qi[x] > 0) landed = mbar_wait_sleep(smem_u32(&q_full[x]), (qi[x] - 1) & 1, 100);
                for (int j = g > F2_KS ? g - F2_KS : 0; j < g && landed; ++j) landed = mbar_wait_sleep(smem_u32(&k_full[j % F2_KS]), (j / F2_KS) & 1, 100);
                for (int j = g > F2_VS ? g - F2_VS : 0; j < g && landed; ++j) landed = mbar_wait_sleep(smem_u32(&v_full[j % F2_VS]), (j / F2_VS) & 1, 100);
                if (ok && !landed) atomicExch(p.err, kDevErrDrain);
            }
        } else if (warp == F2_MMA) {
            constexpr uint32_t idesc_s = idesc_16(FA_M, FA_N, BF16), idesc_o = idesc_16(FA_M, D, BF16) | (1u << 16);  // V is N-major
            bool ok = true;
            int g = 0, gx[2] = {0, 0}, qi[2] = {0, 0};  // key tiles; products of either query tile; items of either
            auto wait = [&](uint64_t *bar, int phase) {
                if (ok && !__all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(bar), phase & 1))) ok = false;
                return ok;
            };
            for (int rd = 0; rd * (int)gridDim.x < items && ok; ++rd) {
                const int w = item_of_round(rd);
                if (w >= items) continue;
                int q0, head, batch, nt[2];
                item_at(w, q0, head, batch, nt);
                const int n = max(nt[0], nt[1]);
                // S(x) = Q(x) K(t)^T; after the last one Q(x) is free.  (Tile 1 finds what tile 0 has waited for.)
                auto scores = [&](int x, int t) {
                    const int s = (g + t) % F2_KS;
                    const uint64_t q_desc = smem_desc_k128(smem_u32(sm_q + x * Cfg::kTile)), k_desc = smem_desc_k128(smem_u32(sm_k + (size_t)s * Cfg::kTile));
                    if (t == 0) wait(&q_full[x], qi[x]);
                    if ((x == 0 || t >= nt[0]) && !wait(&k_full[s], (g + t) / F2_KS)) return;
                    tc_fence_after();
                    if (elect_one()) {
#pragma unroll
                        for (int c = 0; c < SLABS; ++c)
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk)
                                tc_mma_f16(tmem_base + Cfg::kColS + (uint32_t)(x * FA_N), q_desc + (uint64_t)(c * (FA_M * 128 / 16) + kk * 2),
                                           k_desc + (uint64_t)(c * (FA_N * 128 / 16) + kk * 2), idesc_s, (c | kk) != 0);
                        tc_commit(smem_u32(&s_full[x]));
                        if (t == nt[x] - 1) tc_commit(smem_u32(&q_empty[x]));
                    }
                    __syncwarp();
                };
                // O(x) += P(x) V(t), or = at the item's first key tile, when the rows of the item before have left
                auto product = [&](int x, int t) {
                    const int s = (g + t) % F2_VS;
                    const uint64_t v_desc = smem_desc_mn128(smem_u32(sm_v + (size_t)s * Cfg::kTile), FA_N * 128);
                    if (t == 0 && qi[x] >= 1) wait(&o_free[x], qi[x] - 1);
                    if (x == 0 || t >= nt[0]) wait(&v_full[s], (g + t) / F2_VS);
                    if (!wait(&p_full[x], gx[x])) return;
                    tc_fence_after();
                    if (elect_one()) {
#pragma unroll
                        for (int kk = 0; kk < 8; ++kk)  // 16 keys a step: 8 columns of P, 16 rows of 128 bytes of V
                            tc_mma_f16_ts(tmem_base + Cfg::kColO + (uint32_t)(x * D), tmem_base + Cfg::kColS + (uint32_t)(x * FA_N + kk * 8),
                                          v_desc + (uint64_t)(kk * (2048 / 16)), idesc_o, (t | kk) != 0);
                        tc_commit(smem_u32(&o_done[x]));
                    }
                    __syncwarp();
                    ++gx[x];
                };
                auto free_after = [&](uint64_t *bar) {
                    if (ok && elect_one()) tc_commit(smem_u32(bar));
                    __syncwarp();
                };
                if (nt[0] > 0) scores(0, 0);
                if (nt[1] > 0 && ok) scores(1, 0);
                if (n > 0 && ok) free_after(&k_empty[g % F2_KS]);
                for (int t = 0; t < n && ok; ++t) {
                    if (t < nt[0]) {
                        product(0, t);
                        if (t + 1 < nt[0] && ok) scores(0, t + 1);
                    }
                    if (t < nt[1] && ok) product(1, t);
                    if (ok) free_after(&v_empty[(g + t) % F2_VS]);
                    if (t + 1 < nt[1] && ok) scores(1, t + 1);
                    if (t + 1 < n && ok) free_after(&k_empty[(g + t + 1) % F2_KS]);
                }
                g += n;
                qi[0] += nt[0] > 0, qi[1] += nt[1] > 0;
            }
            if (!ok && lane == 0) atomicExch(p.err, kDevErrMma);
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(F2_REGS_SOFTMAX));
        constexpr int HC = FA_N / 2, HD = D / 2;
        const int x = (warp - F2_SOFTMAX) >> 3, half = ((warp - F2_SOFTMAX) >> 2) & 1, quarter = warp & 3, r = quarter * 32 + lane, pair = 1 + x * 4 + quarter;
        const uint32_t lanes = tmem_base + ((uint32_t)(quarter * 32) << 16);
        const uint32_t s_addr = lanes + Cfg::kColS + (uint32_t)(x * FA_N + half * HC), p_addr = lanes + Cfg::kColS + (uint32_t)(x * FA_N + half * (HC / 2));
        const uint32_t o_addr = lanes + Cfg::kColO + (uint32_t)(x * D + half * HD);
        float *own = sm_half + (x * 2 + half) * FA_M + r, *other = sm_half + (x * 2 + (half ^ 1)) * FA_M + r;
        auto meet = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(pair) : "memory"); };
        // A warp whose wait gives up goes on without waiting, on whatever it finds, so that its partner meets it at the barriers.
        bool ok = true, waited_prior = false;
        auto wait = [&](uint64_t *bar, int phase) {
            if (ok) ok = __all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(bar), phase & 1));
            tc_fence_after();
        };
        int g = 0;
        for (int rd = 0; rd * (int)gridDim.x < items; ++rd) {
            const int w = item_of_round(rd);
            if (w >= items) continue;
            int q0, head, batch, nt[2];
            item_at(w, q0, head, batch, nt);
            const int n = nt[x], row = q0 + x * FA_M + r;              // global query index
            const int causal_lim = p.causal ? row + off : 0x7FFFFFFF;  // last visible key
            float m = -INFINITY;                                       // the row's maximum so far (raw scores)
            float l = 0.0f;                                            // sum of this half
            for (int t = 0; t < n; ++t, ++g) {
                wait(&s_full[x], g);
                const int kmax = min(p.seqlen_k - 1, causal_lim) - t * FA_N - half * HC;  // columns > kmax of this half are masked
                const bool cut = !__all_sync(0xffffffffu, kmax >= HC - 1);
                uint32_t sv[HC];
#pragma unroll
                for (int c = 0; c < HC / 32; ++c) tmem_ld32_async(s_addr + c * 32, sv + c * 32);
                tmem_wait_ld();
                if (cut)
#pragma unroll
                    for (int i = 0; i < HC; ++i) sv[i] = i <= kmax ? sv[i] : 0xFF800000u;
                // the row's maximum so far (the partner's half through shared memory: it has read this word's last value before
                // its part of the last P was handed over, and these scores were computed after that)
                float m4[4];  // independent chains
#pragma unroll
                for (int u = 0; u < 4; ++u) m4[u] = __uint_as_float(sv[u]);
#pragma unroll
                for (int i = 4; i + 8 <= HC; i += 8) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) m4[u] = max3(m4[u], __uint_as_float(sv[i + u]), __uint_as_float(sv[i + 4 + u]));
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) m4[u] = fmaxf(m4[u], __uint_as_float(sv[HC - 4 + u]));
                const float m_half = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
                *own = m_half;
                meet();  // (needed for P as well, which goes where the other half's scores were)
                const float m_new = max3(m, m_half, *other), m_use = m_new == -INFINITY ? 0.0f : m_new;  // (nothing to see yet: every p is 0)
                const float alpha = fast_ex2((m - m_use) * p.scale_log2);  // m = -inf gives 0
                m = m_new;
                // p = exp2(s * scale_log2 - m * scale_log2), summed in f32, as 16-bit pairs.  Every third pair takes the f32
                // pipes, which have less to do than the special-function unit with its 16 lanes a cycle and SM.
                const uint64_t c2 = dup2(p.scale_log2), mb2 = dup2(-m_use * p.scale_log2);
                uint64_t sum[2] = {0, 0};
                uint32_t pk[HC / 2];
#pragma unroll
                for (int i = 0; i < HC / 2; ++i) {
                    const uint64_t x2 = fma2(pack2(__uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1])), c2, mb2);
                    float e0, e1;
                    if (i % 3 == 2) {
                        unpack2(ex2_poly2(x2), e0, e1);
                    } else {
                        unpack2(x2, e0, e1);
                        e0 = fast_ex2(e0), e1 = fast_ex2(e1);
                    }
                    sum[i & 1] = add2(sum[i & 1], pack2(e0, e1));
                    pk[i] = pack16<BF16>(e0, e1);
                }
                tmem_st32(p_addr, pk);
                float a, b;
                unpack2(add2(sum[0], sum[1]), a, b);
                l = fmaf(l, alpha, a + b);
                // The products so far are complete: the scores above were issued behind them.
                if (t > 0 && __any_sync(0xffffffffu, alpha != 1.0f)) {
                    const uint64_t alpha2 = dup2(alpha);
#pragma unroll
                    for (int c = 0; c < HD / 32; ++c) {
                        uint32_t o[32];
                        tmem_ld32_async(o_addr + c * 32, o);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            float lo, hi;
                            unpack2(mul2(pack2(__uint_as_float(o[2 * i]), __uint_as_float(o[2 * i + 1])), alpha2), lo, hi);
                            o[2 * i] = __float_as_uint(lo), o[2 * i + 1] = __float_as_uint(hi);
                        }
                        tmem_st32(o_addr + c * 32, o);
                    }
                }
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&p_full[x]));  // this warp's part of P is in place
            }
            if (!waited_prior) {
                pdl_wait_prior();  // the output buffers may still be read by an earlier kernel
                waited_prior = true;
            }
            if (n > 0) {
                meet();  // the partner has read the last maximum
                *own = l;
                meet();
                l += *other;
                meet();  // the next item's maxima go to the same words, and its scores do not wait for the partner's read
            }
            if (half == 0 && p.lse && row < p.seqlen_q)  // kernels/softmax.h:206: max * scale + log(sum); +inf for a row with nothing to attend to
                p.lse[((int64_t)batch * p.h + head) * p.seqlen_q + row] = (l == 0.0f || l != l) ? INFINITY : m * p.scale + logf(l);
            uint16_t *dst = reinterpret_cast<uint16_t *>(p.o) + (int64_t)batch * p.o_batch_stride + (int64_t)row * p.o_row_stride + (int64_t)head * p.o_head_stride + half * HD;
            uint32_t o[HD];
            if (n > 0) {
                wait(&o_done[x], g - 1);
#pragma unroll
                for (int c = 0; c < HD / 32; ++c) tmem_ld32_async(o_addr + c * 32, o + c * 32);
                tmem_wait_ld();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&o_free[x]));
            } else {  // nothing to attend to: zeros, as the reference writes
#pragma unroll
                for (int c = 0; c < HD; ++c) o[c] = 0;
            }
            if (ok && row < p.seqlen_q) {
                const float inv = l > 0.0f ? 1.0f / l : 0.0f;
#pragma unroll
                for (int c = 0; c < HD / 8; ++c) {
                    uint4 wv;
                    wv.x = pack16<BF16>(__uint_as_float(o[8 * c]) * inv, __uint_as_float(o[8 * c + 1]) * inv);
                    wv.y = pack16<BF16>(__uint_as_float(o[8 * c + 2]) * inv, __uint_as_float(o[8 * c + 3]) * inv);
                    wv.z = pack16<BF16>(__uint_as_float(o[8 * c + 4]) * inv, __uint_as_float(o[8 * c + 5]) * inv);
                    wv.w = pack16<BF16>(__uint_as_float(o[8 * c + 6]) * inv, __uint_as_float(o[8 * c + 7]) * inv);
                    reinterpret_cast<uint4 *>(dst)[c] = wv;
                }
            }
            __syncwarp();
        }
        if (!ok && lane == 0) atomicExch(p.err, kDevErrFullWait);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == F2_MMA) tmem_dealloc(tmem_base, 512);
}

template <int D, bool BF16>
cq_status run_two_tiles(cq_ctx *ctx, const CUtensorMap &tq, const CUtensorMap &tk, const CUtensorMap &tv, const FaParams &p) {
    static thread_local int configured = -1;
    if (configured != ctx->device) {
        cudaFuncAttributes fa;
        CQ_CUDA(ctx, cudaFuncGetAttributes(&fa, fmha_two_tiles_kernel<D, BF16>));
        if (fa.numRegs < F2_REGS_LAUNCH) return cq_fail(ctx, CQ_ERR_CUDA, "flash attention: built with fewer registers than its warps divide up");
        CQ_CUDA(ctx, cudaFuncSetAttribute(fmha_two_tiles_kernel<D, BF16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)F2Cfg<D>::kSmem));
        configured = ctx->device;
    }
    const int64_t items = (int64_t)((p.seqlen_q + 2 * FA_M - 1) / (2 * FA_M)) * p.h * p.b;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(items < ctx->sm_count ? items : ctx->sm_count));
    cfg.blockDim = dim3(F2_THREADS);
    cfg.dynamicSmemBytes = F2Cfg<D>::kSmem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ctx->tune.pdl ? 1 : 0;
    CQ_CUDA(ctx, cudaLaunchKernelEx(&cfg, fmha_two_tiles_kernel<D, BF16>, tq, tk, tv, p));
    return CQ_OK;
}

}  // namespace

cq_status launch_fmha_two_tiles(cq_ctx *ctx, const CUtensorMap &tq, const CUtensorMap &tk, const CUtensorMap &tv, const FaParams &p, int d, bool bf16) {
    if (d == 128) return bf16 ? run_two_tiles<128, true>(ctx, tq, tk, tv, p) : run_two_tiles<128, false>(ctx, tq, tk, tv, p);
    return bf16 ? run_two_tiles<64, true>(ctx, tq, tk, tv, p) : run_two_tiles<64, false>(ctx, tq, tk, tv, p);
}
