// CQ_ACT_Q8_1 batches, Y[m,n] = X[m,k] . W[n,k]^T for Q4_0 / Q8_0 weights, with f16 products per weight block:
//
//   y[c, r] = s_c * sum over blocks b of  d[r, b] * ( sum over the block's 32 values of q[r, i] * (hi[c, i] + lo[c, i]) )
//
// q: the block's whole numbers, exact in f16.  hi + lo: the numbers d8 * q8 that quantize_q8_1 makes of an activation row
// (quantized.cu:3521-3558), 19 bits; scaled by a power of two so that the row's largest value sits just below 2^15 the sum of
// two f16 numbers holds them exactly, whatever a block's size beside its row's: d8 is an f16 number, so the values are multiples
// of 2^-24 before that scaling, and lo is kept times 2^11.  Each block's dots are a product of their own in a rotating slot of
// tensor memory, two K = 16 steps with lo, then two with hi, the first of which takes the accumulator times 2^-11 (lo first: the
// tensor core truncates when it adds, and so it does on the small numbers); the epilogue multiplies by d and adds up in f32
// registers, one fused multiply-add per result.  Against Q4_0 a block's dot is sumi d8 - 8 s8 with the block's sum s8 in f16
// (vec_dot_q4_0_q8_1, :1919-1941), which differs from sum (q - 8) d8 q8 by c = 8 (sum d8 q8 - s8): a fifth K = 16 step between
// the two multiplies (c_hi, c_lo 2^11) / 512 by (512, 1/4).
//
// The int8 GEMM (gemm_i8_tmem.cu), which served these batches and still serves the small ones, has exact whole-number dots but
// scales them by both operands' block scales in the epilogue, and an activation scale, the same in every lane, costs a warp
// as much to fetch from shared memory as 32 different values.  us at n 11008 x k 4096, calls back to back, Q4_0 / Q8_0, before ->
// now: 64 rows 45 / 37 -> 32 / 30, 100 rows 73 / 63 -> 39 / 37, 300 rows 217 / 188 -> 85 / 81.
// What bounds it: the way of a slot round the ring (MMAs, commit, poll, tensor-memory load, arrive, poll: about 1500 cycles),
// three slots under way; the tensor pipe is active in 57 / 48 % of the cycles, the issue slots in 55 % (100 rows, n 32000).  Measured on 512 rows of the same kernel in f32 arithmetic: sixteen
// epilogue warps of 32 columns 107, eight of 64 103; sleeping polls 122; one issuing warp instead of two 111; on CTA pairs
// (half the activation traffic, but barriers across the pair) 99 with sixteen warps.
//
// A CTA works on 128 weight rows x NB batch rows:
//   warp 0     TMA, X slabs of 64 k (a unit: two blocks)
//   warp 1     TMA, raw blocks: [128 rows x 144 / 272 B] per 256 k
//   warps 2,3  MMA issue, alternate slots; the whole warp runs the loop, one lane issues
//   warps 4-11 two groups of four: raw blocks -> f16 whole numbers in tensor memory (A operand, four buffers of a unit), the
//              blocks' scales into a ring in shared memory
//   warps 12+  eight epilogue warps: lane = weight row, two warps per 32 rows take half of the columns each
// Slots are 128 columns: one block of 128 batch rows or two of 64, handed over by one commit and one barrier round.
// The epilogue takes registers from the other warps (setmaxnreg).
// Work is the list of (tile, 256-wide chunk of k), cut into equal contiguous shares per CTA; partial tiles go to scratch and
// a small kernel adds them in order (the same bits from run to run).  Every wait is bounded.
//
// Left to the epilogue warps, behind all other work of the CTA, when nobody waits for them: weight rows with an infinite or NaN scale,
// and activation rows with a d8 or s8 that f16 does not hold (values beyond 8.3e6, blocks that sum up to 65520; the pre-pass hands
// over a negative scale).  None of their results is finite, and the blocks concerned alone say which infinity or NaN each is.
#include <type_traits>

#include "gemm_raw.cuh"

namespace {

constexpr int GB_SLOTS = 3;    // of 128 tensor-memory columns
constexpr int GB_EPW = 8;      // epilogue warps
constexpr int GB_SCALES = 8;   // units in the ring of weight scales (see the kernel)
constexpr int GB_A = 4;        // A buffers of 32 tensor-memory columns (a unit)
constexpr int GB_LO_BITS = 11; // lo is kept times 2^11
constexpr float GB_LO = 1 << GB_LO_BITS;
constexpr int GB_LIST = 8192;  // blocks of a row looked over at a time for what is not finite

template <int QT, int NB>
struct GbCfg {
    static constexpr bool kFix = QT == CQ_Q4_0;                // the fifth step
    static constexpr int kBlockBytes = QT == CQ_Q4_0 ? kQ4Bytes : kQ8Bytes;
    static constexpr int kRowChunk = 8 * kBlockBytes;          // 144 / 272 bytes
    static constexpr int kWBytes = GP_ROWS * kRowChunk;
    static constexpr int kWStages = QT == CQ_Q4_0 ? 3 : 2;
    static constexpr int kBoxBytes = NB * 128;                 // 64 k of the batch rows
    static constexpr int kXBytes = 2 * kBoxBytes;              // hi, lo
    static constexpr int kXStages = 4;                         // a chunk's units: its first one, with the corrections, is always in stage 0
    static constexpr int kFixBytes = kFix ? NB * 64 : 0;       // a chunk's corrections, two buffers
    static constexpr int kOnesBytes = kFix ? GP_ROWS * 128 : 0;
    static constexpr int kScaleBytes = GB_SCALES * GP_ROWS * 4;
    static constexpr int kWarpDq0 = 4, kWarpEp0 = 12;
    static constexpr int kThreads = 32 * (kWarpEp0 + GB_EPW);
    static constexpr int kBars = 2 * kWStages + 2 * kXStages + GB_A + 2 * GB_SLOTS;
    static constexpr size_t kSmem = (size_t)kXStages * kXBytes + 2 * kFixBytes + kOnesBytes + (size_t)kWStages * kWBytes + kScaleBytes + 1024 + 8 * kBars + 16;
    static constexpr int kACol0 = 128 * GB_SLOTS;
    static_assert(kSmem <= 232448 && kACol0 + 32 * GB_A <= 512, "shared / tensor memory");
    static_assert(kXStages * kXBytes >= 4 * (GB_LIST + 129), "room for a list of blocks");
};

// What quantize_q8_1 makes of a value (true division, ties away from zero).
__device__ __forceinline__ float gb_q8(float v, float d) { return (float)(int)roundf(__fdiv_rn(v, d)); }

// One CTA per row: largest magnitude, then d8 q8 2^e = hi + lo 2^-11 with 2^14 <= amax 2^e < 2^15 (e = 0 for a row of zeros).
// Exact: d8 q8 has 18 bits and is a multiple of 2^-24, and where d8 is finite (amax < 2^23) e is at least -8, so lo 2^11 is a
// multiple of 2^-21; a d8 below f16's normal numbers is up to twice amax / 127 and leaves hi below 65024 and lo 2^11 below 2^15.
// A row with a d8 or s8 that is not finite gets a negative scale, which leaves it to the epilogue warps.
// fix: [m][k / 8], per 128 k the four blocks' (c_hi, c_lo 2^11) and eight zeros.
__global__ void __launch_bounds__(1024) gb_x_q8_kernel(const float *__restrict__ x, int64_t k, int64_t ldx, int order, __half *__restrict__ hi,
                                                       __half *__restrict__ lo, __half *__restrict__ fix, float *__restrict__ scale) {
    pdl_launch_dependents();
    pdl_wait_prior();
    __shared__ float red[32];
    const int threads = blockDim.x;
    const int64_t row = blockIdx.x;
    const float *src = x + row * ldx;
    const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0 && ldx % 4 == 0;
    float amax = 0.0f;
    if (vec) {
#pragma unroll 4
        for (int64_t i = threadIdx.x; i < k / 4; i += threads) {
            const float4 t = reinterpret_cast<const float4 *>(src)[i];
            amax = fmaxf(amax, fmaxf(fmaxf(fabsf(t.x), fabsf(t.y)), fmaxf(fabsf(t.z), fabsf(t.w))));
        }
    } else {
        for (int64_t i = threadIdx.x; i < k; i += threads) amax = fmaxf(amax, fabsf(src[i]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
    __syncthreads();
    amax = red[0];
    for (int i = 0; i < threads / 32; i += 8)
#pragma unroll
        for (int j = 0; j < 8; ++j) amax = fmaxf(amax, red[i + j]);
    int e = 0;
    if (amax > 0.0f && amax < INFINITY) e = min(14 - ilogbf(amax), 126);
    const float up = __int_as_float((127 + e) << 23);  // e in [-113, 126]
    bool odd = false;
#pragma unroll 4
    for (int64_t o8 = threadIdx.x; o8 < k / 8; o8 += threads) {
        float v[8];
        load_permuted8(src + (o8 >> 2) * 32, (int)(o8 & 3), order, vec, v);
        // a block's 32 values lie in four neighbouring lanes (k is a multiple of 256: warps are in the loop as a whole)
        float top = fmaxf(fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))), fmaxf(fmaxf(fabsf(v[4]), fabsf(v[5])), fmaxf(fabsf(v[6]), fabsf(v[7]))));
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
        const float d = __fdiv_rn(top, 127.0f), dh = __half2float(__float2half_rn(d));
        float q[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) q[j] = top == 0.0f ? 0.0f : gb_q8(v[j], d);
        if (fix) {
            // The block's sum along the reference's xor butterfly (offsets 16, 8, 4, 2, 1).  Lane c of a block holds
            // values 8c .. (order 0: pairs (0,4)(1,5)(2,6)(3,7)) or 4c .. and 16 + 4c .. (order 1: (0,2)(16,18)(1,3)(17,19)).
            float s;
            if (order == 0) {
                float t[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    t[j] = __fadd_rn(v[j], __shfl_xor_sync(0xffffffffu, v[j], 2));
                    t[j] = __fadd_rn(t[j], __shfl_xor_sync(0xffffffffu, t[j], 1));
                }
                const float a0 = __fadd_rn(t[0], t[1]), a1 = __fadd_rn(t[2], t[3]), a2 = __fadd_rn(t[4], t[5]), a3 = __fadd_rn(t[6], t[7]);
                s = __fadd_rn(__fadd_rn(a0, a2), __fadd_rn(a1, a3));
            } else {
                float t[4] = {__fadd_rn(v[0], v[2]), __fadd_rn(v[4], v[6]), __fadd_rn(v[1], v[3]), __fadd_rn(v[5], v[7])};  // values 4c .. 4c + 3, plus 16 further
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    t[j] = __fadd_rn(t[j], __shfl_xor_sync(0xffffffffu, t[j], 2));
                    t[j] = __fadd_rn(t[j], __shfl_xor_sync(0xffffffffu, t[j], 1));
                }
                s = __fadd_rn(__fadd_rn(t[0], t[2]), __fadd_rn(t[1], t[3]));
            }
            float qs = ((q[0] + q[1]) + (q[2] + q[3])) + ((q[4] + q[5]) + (q[6] + q[7]));  // whole numbers
            qs += __shfl_xor_sync(0xffffffffu, qs, 1);
            qs += __shfl_xor_sync(0xffffffffu, qs, 2);
            const float sh = __half2float(__float2half_rn(s)), c = __fsub_rn(8.0f * (dh * qs), 8.0f * sh) * up * 0x1p-9f;
            odd |= !(fabsf(c) < 65000.0f);  // an infinite s8, or a NaN one (with a d8 below f16's normal numbers c reaches 768 amax 2^e / 512, 49152)
            const int64_t blk = o8 >> 2;
            __half *dst = fix + row * (k / 8) + (blk >> 2) * 16;
            if ((o8 & 3) == 0) {
                const __half ch = __float2half_rn(c);
                *reinterpret_cast<__half2 *>(dst + 2 * (blk & 3)) = __halves2half2(ch, __float2half_rn((c - __half2float(ch)) * GB_LO));
            } else if ((o8 & 3) == 1) {
                *reinterpret_cast<uint32_t *>(dst + 8 + 2 * (blk & 3)) = 0;
            }
        }
        odd |= dh == INFINITY;
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = q[j] * dh;
        uint32_t wh[4], wl[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float a = v[2 * j] * up, b = v[2 * j + 1] * up;
            const __half2 h = __floats2half2_rn(a, b);
            const __half2 l = __floats2half2_rn((a - __low2float(h)) * GB_LO, (b - __high2float(h)) * GB_LO);
            wh[j] = *reinterpret_cast<const uint32_t *>(&h);
            wl[j] = *reinterpret_cast<const uint32_t *>(&l);
        }
        *reinterpret_cast<uint4 *>(hi + row * k + o8 * 8) = make_uint4(wh[0], wh[1], wh[2], wh[3]);
        *reinterpret_cast<uint4 *>(lo + row * k + o8 * 8) = make_uint4(wl[0], wl[1], wl[2], wl[3]);
    }
    odd = __syncthreads_or(odd);
    if (threadIdx.x == 0) scale[row] = (odd ? -1.0f : 1.0f) * __int_as_float((127 - e) << 23);
}

// Results that are not finite.  A weight row with an infinite or NaN scale, or an activation row with such a d8 or s8, has none that
// are, and its other blocks, whose terms are finite, have no say in which: only the terms of those blocks are added up.

// d8 and s8 of a block of 32 values (16-byte aligned) as the reference computes them, before their rounding to f16.
__device__ __forceinline__ void gb_block_scales(const float *xb, float &d8, float &s8) {
    float s[16], top = 0.0f;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const float4 f = reinterpret_cast<const float4 *>(xb)[u], g = reinterpret_cast<const float4 *>(xb)[4 + u];
        top = fmaxf(top, fmaxf(fmaxf(fmaxf(fabsf(f.x), fabsf(f.y)), fmaxf(fabsf(f.z), fabsf(f.w))), fmaxf(fmaxf(fabsf(g.x), fabsf(g.y)), fmaxf(fabsf(g.z), fabsf(g.w)))));
        s[4 * u] = __fadd_rn(f.x, g.x), s[4 * u + 1] = __fadd_rn(f.y, g.y), s[4 * u + 2] = __fadd_rn(f.z, g.z), s[4 * u + 3] = __fadd_rn(f.w, g.w);
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1)
#pragma unroll
        for (int u = 0; u < o; ++u) s[u] = __fadd_rn(s[u], s[u + o]);
    d8 = __fdiv_rn(top, 127.0f), s8 = s[0];
}
__device__ __forceinline__ bool gb_odd_half(unsigned short h) { return (h & 0x7C00) == 0x7C00; }
template <int QT>
__device__ __forceinline__ bool gb_odd_block(const float *xb) {
    float d8, s8;
    gb_block_scales(xb, d8, s8);
    return gb_odd_half(__half_as_ushort(__float2half_rn(d8))) || (QT == CQ_Q4_0 && gb_odd_half(__half_as_ushort(__float2half_rn(s8))));
}
// A block's term.
template <int QT>
__device__ __noinline__ float gb_term(const uint8_t *block, const float *xb, int order) {
    constexpr int BB = QT == CQ_Q4_0 ? kQ4Bytes : kQ8Bytes;
    const unsigned short *blk = reinterpret_cast<const unsigned short *>(block);
    float d8, s8, dot = 0.0f;
    gb_block_scales(xb, d8, s8);
    auto q8 = [&](int i) { return d8 == 0.0f ? 0.0f : gb_q8(xb[i], d8); };
    for (int j = 0; j < (BB - 2) / 2; ++j) {
        const int two = blk[1 + j];
        if (QT == CQ_Q4_0) {
            for (int h = 0; h < 4; ++h) {  // byte 2j (+1): its low and its high nibble
                const int byte = 2 * j + (h >> 1);
                dot += (float)((two >> (8 * (h >> 1) + 4 * (h & 1))) & 15) * q8(order == CQ_ORDER_GO_INTERLEAVED ? 2 * byte + (h & 1) : byte + 16 * (h & 1));
            }
        } else {
            dot += (float)(signed char)(two & 0xFF) * q8(2 * j) + (float)(signed char)(two >> 8) * q8(2 * j + 1);
        }
    }
    const float d = __half2float(__ushort_as_half(blk[0])), dh = __half2float(__float2half_rn(d8));
    return QT == CQ_Q4_0 ? d * fmaf(dot, dh, -8.0f * __half2float(__float2half_rn(s8))) : d * dh * dot;
}
// Weight rows j0 .. j0 + 127 (below p.n) by batch row c over blocks [b0, b1), the terms of the batch row's blocks that are not
// finite: the 256 epilogue threads (t) together.  out[j] = (bias +) their sum.  `list`: GB_LIST + 129 words.
template <int QT>
__device__ __noinline__ void gb_odd_row(const GpParams &p, int j0, int c, int b0, int b1, int *list, float *out, bool bias, int t) {
    constexpr int BB = QT == CQ_Q4_0 ? kQ4Bytes : kQ8Bytes;
    int *count = list + GB_LIST;
    float *sum_s = reinterpret_cast<float *>(count + 1);
    const float *xrow = p.x + (int64_t)c * p.ldx;
    const int r = t & 127, j = j0 + r;
    const uint8_t *wrow = p.w + (int64_t)j * (p.k / kQK) * BB;
    float sum = 0.0f;
    for (int from = b0; from < b1; from += GB_LIST) {
        const int to = min(b1, from + GB_LIST);
        asm volatile("barrier.cta.sync 1, 256;" ::: "memory");  // the list before is done with
        if (t == 0) *count = 0;
        asm volatile("barrier.cta.sync 1, 256;" ::: "memory");
        for (int b = from + t; b < to; b += 256)
            if (gb_odd_block<QT>(xrow + (int64_t)b * kQK)) list[atomicAdd(count, 1)] = b;
        asm volatile("barrier.cta.sync 1, 256;" ::: "memory");
        const int n = *count;
        if (j < p.n)
            for (int i = t >> 7; i < n; i += 2) sum += gb_term<QT>(wrow + (int64_t)list[i] * BB, xrow + (int64_t)list[i] * kQK, p.order);
    }
    if (t >= 128) sum_s[r] = sum;
    asm volatile("barrier.cta.sync 1, 256;" ::: "memory");
    if (t < 128 && j < p.n) out[r] = (bias ? p.bias[j] : 0.0f) + (sum + sum_s[r]);
}
// Weight row j by batch rows c0 .. c0 + columns - 1 over blocks [b0, b1), the terms of the weight row's blocks whose scale is not
// finite: a warp.  Added to what is there for batch rows of the kind above.
template <int QT>
__device__ __noinline__ void gb_odd_weights(const GpParams &p, int j, int c0, int columns, int b0, int b1, float *out, int64_t ld, bool bias, int lane) {
    constexpr int BB = QT == CQ_Q4_0 ? kQ4Bytes : kQ8Bytes;
    const uint8_t *wrow = p.w + (int64_t)j * (p.k / kQK) * BB;
    for (int c = lane; c < columns; c += 32) {
        float sum = 0.0f;
        for (int b = b0; b < b1; ++b)
            if (gb_odd_half(*reinterpret_cast<const unsigned short *>(wrow + (int64_t)b * BB)))
                sum += gb_term<QT>(wrow + (int64_t)b * BB, p.x + (int64_t)(c0 + c) * p.ldx + (int64_t)b * kQK, p.order);
        out[c * ld] = (p.xscale[c0 + c] < 0.0f ? out[c * ld] : bias ? p.bias[j] : 0.0f) + sum;
    }
}
// Whether any of the 256 epilogue threads says so.
__device__ __forceinline__ bool gb_any(bool mine) {
    int any;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, 1, 256, p;\n\tselp.s32 %0, 1, 0, q;\n\t}" : "=r"(any) : "r"((int)mine) : "memory");
    return any;
}

template <int R>
__device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R)); }
template <int R>
__device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R)); }
// What the roles' four, eight and eight warps hold after the split: together no more than 640 threads were launched with.
constexpr int GB_REGS_LAUNCH = 96, GB_REGS_CONTROL = 40, GB_REGS_DQ = 56, GB_REGS_EP = 160;
static_assert(128 * GB_REGS_CONTROL + 256 * GB_REGS_DQ + 256 * GB_REGS_EP <= 640 * GB_REGS_LAUNCH, "registers of the block");

// Descriptor of a K-major tile stored as rows of 64 bytes with the 64-byte swizzle: 8-row atoms 512 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_k64(uint32_t smem_addr) {
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)4 << 61);
}

template <int QT, int NB>
__global__ void __launch_bounds__(GbCfg<QT, NB>::kThreads, 1)
    gemm_blocks_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmFix, const __grid_constant__ GpParams p) {
    using Cfg = GbCfg<QT, NB>;
    constexpr int WST = Cfg::kWStages, XST = Cfg::kXStages, ROWCHUNK = Cfg::kRowChunk;
    constexpr int BPS = 128 / NB;  // blocks per slot: 1, 2
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *smem_x = smem;                                          // XST slabs (1024-byte aligned boxes)
    uint8_t *smem_fix = smem + (size_t)XST * Cfg::kXBytes;
    uint8_t *smem_ones = smem_fix + 2 * Cfg::kFixBytes;              // the fifth step's A operand
    uint8_t *smem_w = smem_ones + Cfg::kOnesBytes;                   // WST raw stages
    uint32_t *smem_d = reinterpret_cast<uint32_t *>(smem_w + (size_t)WST * Cfg::kWBytes);  // [GB_SCALES][128 rows]: a unit's two scales of a row
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem_d + GB_SCALES * GP_ROWS);
    uint64_t *w_full = bars, *w_empty = w_full + WST, *x_full = w_empty + WST, *u_done = x_full + XST, *a_full = u_done + XST, *d_full = a_full + GB_A,
             *d_empty = d_full + GB_SLOTS;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(d_empty + GB_SLOTS);

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int g0 = blockIdx.x * p.per_share, g1 = min(g0 + p.per_share, p.total);
    const int nu = 4 * (g1 - g0);  // units of this share

    if (threadIdx.x == 0) {
        for (int s = 0; s < WST; ++s) {
            mbar_init(smem_u32(&w_full[s]), 1);
            mbar_init(smem_u32(&w_empty[s]), 8);      // the two groups that read a stage
        }
        for (int s = 0; s < XST; ++s) {
            mbar_init(smem_u32(&x_full[s]), 1);
            // the unit's MMAs have read its slab and its A buffer (and where the corrections come with a unit that one of the two
            // issuing warps has no part in, that warp has seen it come: the barrier is never two phases ahead of a wait)
            mbar_init(smem_u32(&u_done[s]), BPS == 1 || (Cfg::kFix && s == 0) ? 2 : 1);
        }
        for (int b = 0; b < GB_A; ++b) mbar_init(smem_u32(&a_full[b]), 4);
        for (int s = 0; s < GB_SLOTS; ++s) {
            mbar_init(smem_u32(&d_full[s]), 1);       // the commit of the warp whose slot it is
            mbar_init(smem_u32(&d_empty[s]), GB_EPW);
        }
        fence_mbar_init();
    }
    if constexpr (Cfg::kFix) {
        // Row r of the K-major tile: K = 16 step j (16-byte pieces 2j, 2j + 1, at piece ^ (r & 7)) has 512 at 2j, 512 * 2^-11 at 2j + 1.
        for (int i = threadIdx.x; i < GP_ROWS * 8; i += Cfg::kThreads) {
            const int r = i >> 3, piece = i & 7, j = piece >> 1;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if ((piece & 1) == 0) (j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w) = 0x34006000u;
            *reinterpret_cast<uint4 *>(smem_ones + r * 128 + ((piece ^ (r & 7)) << 4)) = v;
        }
    }
    fence_proxy_async();
    if (warp == 1) tmem_alloc(smem_u32(tmem_slot), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents();  // not before the tensor memory is ours: a dependent may want some too

    if (warp < Cfg::kWarpDq0) {
        regs_dec<GB_REGS_CONTROL>();
        if (warp == 0) {
            // ---- TMA, X: the batch rows, 64 k per unit ----
            if (lane == 0) {
                pdl_wait_prior();
                bool ok = true;
                int u = 0;
                for (; u < nu; ++u) {
                    const int g = g0 + (u >> 2), tile = g / p.nchunks, c = g - tile * p.nchunks;
                    const int s = u % XST;
                    if (u >= XST && !mbar_wait_bounded(smem_u32(&u_done[s]), ((u / XST) - 1) & 1)) {
                        atomicExch(p.err, kDevErrEmptyWait);
                        ok = false;
                        break;
                    }
                    // (the corrections come with a chunk's first unit: XST = 4, so the chunk before the last is done with)
                    const bool fix = Cfg::kFix && (u & 3) == 0;
                    const uint32_t bar = smem_u32(&x_full[s]);
                    mbar_expect_tx(bar, Cfg::kXBytes + (fix ? Cfg::kFixBytes : 0));
                    const int row = (tile % p.mtiles) * NB;
                    tma_load_4d(smem_u32(smem_x + (size_t)s * Cfg::kXBytes), &tmX, 0, row, 4 * c + (u & 3), 0, bar);
                    if (fix) tma_load_2d(smem_u32(smem_fix + ((u >> 2) & 1) * Cfg::kFixBytes), &tmFix, c * 32, row, bar);
                }
                if (ok)  // leave when the last ones have landed
                    for (int j = u > XST ? u - XST : 0; j < u; ++j)
                        if (!mbar_wait_bounded(smem_u32(&x_full[j % XST]), (j / XST) & 1)) {
                            atomicExch(p.err, kDevErrDrain);
                            break;
                        }
            }
        } else if (warp == 1) {
            // ---- TMA, raw blocks of the tile's 128 weight rows, 256 k per stage ----
            if (lane == 0) {
                bool ok = true;
                int i = 0;
                for (; i < nu / 4; ++i) {
                    const int g = g0 + i, tile = g / p.nchunks, c = g - tile * p.nchunks;
                    const int s = i % WST;
                    if (i >= WST && !mbar_wait_bounded(smem_u32(&w_empty[s]), ((i / WST) - 1) & 1)) {
                        atomicExch(p.err, kDevErrEmptyWait);
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(smem_u32(&w_full[s]), Cfg::kWBytes);
                    // rows past n are outside the tensor: zero fill
                    tma_load_2d(smem_u32(smem_w + (size_t)s * Cfg::kWBytes), &tmW, c * (ROWCHUNK / 2), (tile / p.mtiles) * GP_ROWS, smem_u32(&w_full[s]));
                }
                if (ok)
                    for (int j = i > WST ? i - WST : 0; j < i; ++j)
                        if (!mbar_wait_bounded(smem_u32(&w_full[j % WST]), (j / WST) & 1)) {
                            atomicExch(p.err, kDevErrDrain);
                            break;
                        }
            }
        } else {
            // ---- MMA issue: warp e takes every second slot.  (It waits for the reader of slot q - 3 of the other warp, having
            // issued slot q - 2 after the reader of q - 5: the barrier is never two phases behind.) ----
            constexpr uint32_t idesc = idesc_f16(GP_ROWS, NB);
            const int e = warp - 2;
            int slot = 0, use = 0;
            bool ok = true;
            for (int u = 0; u < nu && ok; ++u) {
                const int s = u % XST, b = u % GB_A;
                const uint64_t xh = smem_desc_k128(smem_u32(smem_x + (size_t)s * Cfg::kXBytes)), xl = xh + (uint64_t)(Cfg::kBoxBytes / 16);
                const uint32_t ah = tmem_base + (uint32_t)(Cfg::kACol0 + b * 32);
#pragma unroll
                for (int blk = 0; blk < 2; ++blk) {
                    const bool begins = BPS == 1 || blk == 0, ends = BPS == 1 || blk == 1;
                    const bool mine = (BPS == 1 ? blk : u & 1) == e;
                    if (mine || (Cfg::kFix && blk == 0 && (u & 3) == 0)) {
                        bool there = !begins || mbar_wait_bounded(smem_u32(&x_full[s]), (u / XST) & 1);
                        there = there && (!mine || !begins || mbar_wait_bounded(smem_u32(&a_full[b]), (u / GB_A) & 1));
                        there = there && (!mine || !begins || use == 0 || mbar_wait_bounded(smem_u32(&d_empty[slot]), (use - 1) & 1));
                        if (!__all_sync(0xffffffffu, there)) {
                            if (lane == 0) atomicExch(p.err, kDevErrMma);
                            ok = false;
                            break;
                        }
                        if (BPS == 2 && !mine && lane == 0) mbar_arrive(smem_u32(&u_done[s]));
                    }
                    if (mine) {
                        tc_fence_after();
                        if (elect_one()) {
                            const uint32_t acc = tmem_base + (uint32_t)(slot * 128 + (BPS == 1 ? 0 : blk * NB));
                            tc_mma_f16_ts(acc, ah + 16 * blk, xl + 4 * blk, idesc, 0);
                            tc_mma_f16_ts(acc, ah + 16 * blk + 8, xl + 4 * blk + 2, idesc, 1);
                            if constexpr (Cfg::kFix) {
                                tc_mma_f16_scaled<GB_LO_BITS>(acc, smem_desc_k128(smem_u32(smem_ones)) + (uint64_t)(2 * (2 * (u & 1) + blk)),
                                                              smem_desc_k64(smem_u32(smem_fix + ((u >> 2) & 1) * Cfg::kFixBytes)) + (uint64_t)(2 * ((u >> 1) & 1)), idesc);
                                tc_mma_f16_ts(acc, ah + 16 * blk, xh + 4 * blk, idesc, 1);
                            } else {
                                tc_mma_f16_ts_scaled<GB_LO_BITS>(acc, ah + 16 * blk, xh + 4 * blk, idesc);
                            }
                            tc_mma_f16_ts(acc, ah + 16 * blk + 8, xh + 4 * blk + 2, idesc, 1);
                            if (ends) {
                                tc_commit(smem_u32(&d_full[slot]));
                                tc_commit(smem_u32(&u_done[s]));
                            }
                        }
                        __syncwarp();
                    }
                    if (ends && ++slot == GB_SLOTS) slot = 0, ++use;
                }
            }
        }
    } else if (warp < Cfg::kWarpEp0) {
        // ---- whole numbers of the raw blocks into tensor memory: thread = weight row, group = every second pair of units ----
        regs_dec<GB_REGS_DQ>();
        const int grp = (warp - Cfg::kWarpDq0) >> 2, quarter = warp & 3, r = quarter * 32 + lane;
        const uint32_t a_t = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(Cfg::kACol0 + grp * 64);  // its two A buffers
        auto run = [&](auto which) {
            constexpr int GRP = decltype(which)::value;  // compile-time, so that words stay in registers
            bool ok = true;
            for (int c = 0; c < nu / 4 && ok; ++c) {
                const int s = c % WST;
                if (!mbar_wait_sleep(smem_u32(&w_full[s]), (c / WST) & 1, 20)) {
                    if (lane == 0) atomicExch(p.err, kDevErrFullWait);
                    break;
                }
                // The thread's bytes in 16-byte loads, the only ones that meet no bank twice at a pitch of 144 / 272: Q4_0
                // two units' 72 bytes, Q8_0 68 bytes for each.
                const uint4 *wrow = reinterpret_cast<const uint4 *>(smem_w + (size_t)s * Cfg::kWBytes + r * ROWCHUNK);
                constexpr int PW = ROWCHUNK / 16, VW = (PW - 1) / 2;  // words of two blocks, of a block's values
                uint32_t w[20];
                auto load = [&](int from16) {
#pragma unroll
                    for (int j = 0; j < 5; ++j) {
                        const uint4 t = wrow[from16 + j];
                        w[4 * j] = t.x, w[4 * j + 1] = t.y, w[4 * j + 2] = t.z, w[4 * j + 3] = t.w;
                    }
                };
                if constexpr (QT == CQ_Q4_0) load(GRP * 4);
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                    // Two blocks in PW words: the first starts on a word, its values two bytes in; the second starts two bytes
                    // into the middle word, its values on the next one.
                    constexpr int Q8 = QT == CQ_Q8_0;
                    if (Q8) load((PW * (2 * GRP + hh)) >> 2);
                    const uint32_t *wq = w + (Q8 ? (PW * (2 * GRP + hh)) & 3 : 2 * GRP + PW * hh);
                    const int u = 4 * c + 2 * GRP + hh;
                    if (u >= GB_A && !mbar_wait_sleep(smem_u32(&u_done[(u - GB_A) % XST]), ((u - GB_A) / XST) & 1, 20)) {
                        if (lane == 0) atomicExch(p.err, kDevErrMma);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    // The ring's entry was last used by unit u - 8: the tensor core has done unit u - 4, and it is at most three
                    // slots (three units with 64 batch rows) ahead of the epilogue.
                    smem_d[(u & (GB_SCALES - 1)) * GP_ROWS + r] = __byte_perm(wq[0], wq[VW], 0x7610);
#pragma unroll
                    for (int blk = 0; blk < 2; ++blk) {
                        uint32_t out[16];
#pragma unroll
                        for (int j = 0; j < VW; ++j) {
                            const uint32_t v = blk ? wq[VW + 1 + j] : __funnelshift_r(wq[j], wq[j + 1], 16);
                            if constexpr (QT == CQ_Q4_0) {
                                __half2 q[4];
                                gp_numbers_q4(v, q);
#pragma unroll
                                for (int t = 0; t < 4; ++t) out[4 * j + t] = *reinterpret_cast<const uint32_t *>(&q[t]);
                            } else {
                                __half2 q[2];
                                gp_numbers_q8(v, q);
#pragma unroll
                                for (int t = 0; t < 2; ++t) out[2 * j + t] = *reinterpret_cast<const uint32_t *>(&q[t]);
                            }
                        }
                        tmem_st16(a_t + (uint32_t)(32 * hh + 16 * blk), out);
                    }
                    tmem_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(smem_u32(&a_full[2 * GRP + hh]));
                        // The raw stage is free too: every word of it has gone through a finished store.
                        if (hh == 1) mbar_arrive(smem_u32(&w_empty[s]));
                    }
                }
            }
        };
        if (grp == 0) run(std::integral_constant<int, 0>());
        else run(std::integral_constant<int, 1>());
    } else {
        // ---- epilogue: lane = weight row, two warps per 32 rows take half of the columns each ----
        regs_inc<GB_REGS_EP>();
        pdl_wait_prior();  // y and the partial tiles may still be read by earlier kernels; the row scales are the pre-pass's
        constexpr int COLS = NB / 2;  // of a block; 64 of a slot
        const int quarter = warp & 3, part = (warp - Cfg::kWarpEp0) >> 2, r = quarter * 32 + lane;
        const uint32_t from = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(part * COLS);
        const int first_tile = g0 / p.nchunks;
        int u = 0, slot = 0, use = 0;
        bool ok = true, odd = false, hurt = false;  // (rows that the tensor core does not take, of either operand)
        for (int g = g0; g < g1 && ok;) {
            const int tile = g / p.nchunks, c0 = g - tile * p.nchunks, cn = min(p.nchunks - c0, g1 - g);
            g += cn;
            const int group = tile / p.mtiles, col0 = (tile - group * p.mtiles) * NB + part * COLS;
            uint64_t acc[COLS / 2];
#pragma unroll
            for (int j = 0; j < COLS / 2; ++j) acc[j] = 0;
            for (int e = u + 4 * cn; u < e && ok; ++u) {
                uint32_t two = 0;
#pragma unroll
                for (int gq = 0; gq < 2 / BPS; ++gq) {  // the unit's slots
                    if (!__all_sync(0xffffffffu, mbar_wait_bounded(smem_u32(&d_full[slot]), use & 1))) {
                        if (lane == 0) atomicExch(p.err, kDevErrMma);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    uint32_t v[64];
                    const uint32_t sbase = from + (uint32_t)(slot * 128);
                    tmem_ld32_async(sbase, v);
                    tmem_ld32_async(sbase + (BPS == 1 ? 32 : NB), v + 32);
                    float d[BPS];
#pragma unroll
                    for (int b = 0; b < BPS; ++b) {
                        const int blk = gq * BPS + b;
                        if (blk == 0) {
                            asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(two) : "r"(smem_u32(&smem_d[(u & (GB_SCALES - 1)) * GP_ROWS + r])) : "memory");
                            hurt |= (((two & 0x7C007C00u) + 0x04000400u) & 0x80008000u) != 0;
                        }
                        d[b] = __half2float(__ushort_as_half((unsigned short)(blk ? two >> 16 : two & 0xFFFFu)));
                    }
                    tmem_wait_ld();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&d_empty[slot]));
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        uint64_t &a = acc[j % (COLS / 2)];
                        a = fma2(pack2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])), dup2(d[j / (COLS / 2)]), a);
                    }
                    if (++slot == GB_SLOTS) slot = 0, ++use;
                }
            }
            if (!ok) break;
            const int row = group * GP_ROWS + r;
            // whole k range in this share -> y, otherwise one of this share's two partial tiles
            const bool direct = cn == p.nchunks;
            const int64_t ld = direct ? p.ldy : GP_ROWS;
            float *dst = direct ? p.y + (int64_t)col0 * p.ldy + row
                                : p.part + ((int64_t)(2 * blockIdx.x + (tile == first_tile ? 0 : 1)) * NB + part * COLS) * GP_ROWS + r;
            const float bias = direct && p.bias && row < p.n ? p.bias[row] : 0.0f;
            float scales[COLS / 32];
#pragma unroll
            for (int j = 0; j < COLS / 32; ++j) scales[j] = p.xscale[min(col0 + 32 * j + lane, p.m - 1)];
#pragma unroll
            for (int j = 0; j < COLS / 2; ++j) {
                const float s0 = __shfl_sync(0xffffffffu, scales[j / 16], (2 * j) & 31), s1 = __shfl_sync(0xffffffffu, scales[j / 16], (2 * j + 1) & 31);
                float v0, v1;
                unpack2(acc[j], v0, v1);
                odd |= s0 < 0.0f || s1 < 0.0f;
                if (row < p.n) {
                    if (col0 + 2 * j < p.m) dst[(int64_t)(2 * j) * ld] = fmaf(v0, s0, bias);
                    if (col0 + 2 * j + 1 < p.m) dst[(int64_t)(2 * j + 1) * ld] = fmaf(v1, s1, bias);
                }
            }
            __syncwarp();
        }
        // All units are done with, the slabs of X among them.  (Every one of the 256 threads takes the same way from here.)
        if (gb_any(odd || hurt || !ok) && !gb_any(!ok)) {
            const bool some_hurt = gb_any(hurt);
            const int t = threadIdx.x - 32 * Cfg::kWarpEp0;
            for (int g = g0; g < g1;) {
                const int tile = g / p.nchunks, c0 = g - tile * p.nchunks, cn = min(p.nchunks - c0, g1 - g), b0 = c0 * 8, b1 = (c0 + cn) * 8;
                g += cn;
                const int group = tile / p.mtiles, col0 = (tile - group * p.mtiles) * NB, j0 = group * GP_ROWS, columns = min(NB, p.m - col0);
                const bool direct = cn == p.nchunks;
                const int64_t ld = direct ? p.ldy : GP_ROWS;
                float *out = direct ? p.y + (int64_t)col0 * p.ldy + j0 : p.part + (int64_t)(2 * blockIdx.x + (tile == first_tile ? 0 : 1)) * NB * GP_ROWS;
                for (int c = 0; c < columns; ++c)
                    if (p.xscale[col0 + c] < 0.0f) gb_odd_row<QT>(p, j0, col0 + c, b0, b1, reinterpret_cast<int *>(smem_x), out + c * ld, direct && p.bias, t);
                if (some_hurt) {
                    asm volatile("barrier.cta.sync 1, 256;" ::: "memory");  // the batch rows' sums are there to be added to
                    for (int r = t >> 5; r < GP_ROWS && j0 + r < p.n; r += 8) {
                        bool bad = false;
                        for (int b = b0 + lane; b < b1; b += 32)
                            bad |= gb_odd_half(*reinterpret_cast<const unsigned short *>(p.w + ((int64_t)(j0 + r) * (p.k / kQK) + b) * Cfg::kBlockBytes));
                        if (__any_sync(0xffffffffu, bad)) gb_odd_weights<QT>(p, j0 + r, col0, columns, b0, b1, out + r, ld, direct && p.bias, lane);
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, 512);
}

// The corrections [m][k / 8] of f16, box = 32 values (a chunk) x rows.
bool gb_fix_map(CUtensorMap *map, const void *fix, int64_t m, int64_t k, int rows) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)(k / 8), (cuuint64_t)m};
    cuuint64_t strides[1] = {(cuuint64_t)(k / 8) * 2};
    cuuint32_t box[2] = {32u, (cuuint32_t)rows};
    cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(fix), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int QT, int NB>
cq_status gb_run(cq_ctx *ctx, const float *x, int64_t m, int64_t k, int64_t ldx, int order, const void *w, int64_t n, float *y, int64_t ldy) {
    using Cfg = GbCfg<QT, NB>;
    auto kern = gemm_blocks_kernel<QT, NB>;
    static thread_local int configured = -1;
    if (configured != ctx->device) {
        cudaFuncAttributes fa;
        CQ_CUDA(ctx, cudaFuncGetAttributes(&fa, kern));
        // the roles' registers are shares of what the block was launched with
        if (fa.numRegs < GB_REGS_LAUNCH) return cq_fail(ctx, CQ_ERR_CUDA, "gemm: built with fewer registers than its warps divide up");
        CQ_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::kSmem));
        configured = ctx->device;
    }
    GpParams p = {};
    p.y = y, p.ldy = ldy, p.m = (int)m, p.n = (int)n, p.k = (int)k, p.err = ctx->dev_err_devptr, p.bias = ctx->bias;
    p.x = x, p.w = static_cast<const uint8_t *>(w), p.ldx = ldx, p.order = order;
    const auto up = [](size_t v) { return (v + 1023) & ~size_t(1023); };
    const size_t x_bytes = up((size_t)m * k * 2), fix_bytes = Cfg::kFix ? up((size_t)m * (k / 8) * 2) : 0, scale_bytes = up((size_t)m * 4);
    const size_t operand_bytes = 2 * x_bytes + fix_bytes + scale_bytes;
    GpShares sh;
    cq_status s = gp_share_out(ctx, p, GP_ROWS, NB, ctx->sm_count, operand_bytes, sh);
    if (s != CQ_OK) return s;
    s = cq_reserve_scratch(ctx, operand_bytes + sh.part_bytes);
    if (s != CQ_OK) return s;
    uint8_t *base = static_cast<uint8_t *>(ctx->scratch);
    __half *xh = reinterpret_cast<__half *>(base), *xl = reinterpret_cast<__half *>(base + x_bytes);
    __half *fix = Cfg::kFix ? reinterpret_cast<__half *>(base + 2 * x_bytes) : nullptr;
    float *scale = reinterpret_cast<float *>(base + 2 * x_bytes + fix_bytes);
    p.part = reinterpret_cast<float *>(base + operand_bytes);
    p.xscale = scale;
    CUtensorMap tmW, tmX, tmFix = {};
    if (!gp_w_map(&tmW, w, n, (k / kQK) * Cfg::kBlockBytes, Cfg::kRowChunk) || !gp_x_map(&tmX, xh, m, k, x_bytes, NB, 1) ||
        (Cfg::kFix && !gb_fix_map(&tmFix, fix, m, k, NB)))
        return cq_fail(ctx, CQ_ERR_CUDA, "gemm: cuTensorMapEncodeTiled failed or is unavailable");
    // Threads per row of the pre-pass: where its CTAs have an SM each or share it with one other, a long row wants more than 256.
    // (us of the call at n 700, Q4_0, 256 / 512 / 1024 threads: 64 rows of 4096 values 15.5 / 14.7 / 14.0, of 14336 32.4 / 27.1 /
    // 21.4; 200 rows of 2048 18.2 / 16.5 / 19.6, of 14336 39.9 / 37.6 / 39.5; 400 rows of 4096 27.7 / 29.1 / 32.3.)
    const int threads = m <= ctx->sm_count && k >= 8192 ? 1024 : (m <= 2 * ctx->sm_count && k >= 2048 ? 512 : 256);
    s = gp_launch(ctx, gb_x_q8_kernel, dim3((unsigned)m), threads, 0, false, x, k, ldx, QT == CQ_Q4_0 ? order : 2, xh, xl, fix, scale);
    if (s == CQ_OK) s = gp_launch(ctx, kern, dim3(sh.shares), Cfg::kThreads, Cfg::kSmem, false, tmW, tmX, tmFix, p);
    if (s == CQ_OK && sh.cut) s = gp_launch(ctx, gp_sum_kernel<GP_ROWS, NB>, dim3((unsigned)sh.tiles, NB / 8), 256, 0, false, p);
    if (s == CQ_OK && p.bias) ctx->bias_done = true;
    return s;
}

}  // namespace

cq_status launch_gemm_blocks(cq_ctx *ctx, int qtype, int order, const float *x, int64_t m, int64_t k, int64_t ldx, const void *w, int64_t n, float *y,
                             int64_t ldy) {
    if ((reinterpret_cast<uintptr_t>(x) & 3) != 0 || (reinterpret_cast<uintptr_t>(y) & 3) != 0)
        return cq_fail(ctx, CQ_ERR_INVALID_ARG, "gemm: misaligned pointer");
    if (qtype == CQ_Q4_0)
        return m <= 64 ? gb_run<CQ_Q4_0, 64>(ctx, x, m, k, ldx, order, w, n, y, ldy) : gb_run<CQ_Q4_0, 128>(ctx, x, m, k, ldx, order, w, n, y, ldy);
    return m <= 64 ? gb_run<CQ_Q8_0, 64>(ctx, x, m, k, ldx, order, w, n, y, ldy) : gb_run<CQ_Q8_0, 128>(ctx, x, m, k, ldx, order, w, n, y, ldy);
}
