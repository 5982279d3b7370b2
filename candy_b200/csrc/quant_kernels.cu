// Block-format conversion kernels: blocks -> f32 (bit-exact), f32 -> Q4_0 / Q8_0 weight
// blocks, f32 -> Q8_1 activation blocks.  All are streaming, HBM-bound kernels; none is
// on the per-token hot path (weights are quantized once, dequantize is a utility).
#include "common.cuh"

namespace {

__device__ __forceinline__ uint32_t ld_u16(const uint8_t *p) { return *reinterpret_cast<const unsigned short *>(p); }

// d * f with the NaN bit patterns the reference's CPU path produces on amd64 (SSE MULSS):
// a NaN scale comes back quieted with its payload, inf * 0 gives the default NaN 0xFFC00000.
// The GPU multiplier would return the canonical 0x7FFFFFFF for both.
__device__ __forceinline__ float mul_like_cpu(float d, float f) {
    float r = __fmul_rn(d, f);
    if (r != r) {
        const uint32_t db = __float_as_uint(d);
        r = ((db & 0x7FFFFFFFu) > 0x7F800000u) ? __uint_as_float(db | 0x00400000u) : __uint_as_float(0xFFC00000u);
    }
    return r;
}

// One thread produces four consecutive f32 values (one 16-byte store), so a warp writes
// 512 contiguous bytes.  Semantics: tensor/internal/cpu/kernels/quantized.go:85-93
// (ORDER 0), tensor/internal/cuda/kernels/quantized.cu:838-867 (ORDER 1), quantized.go:
// 131-136 (Q8_0).  d*(q-8) and d*q are exact in f32, so the results are bit-identical to
// the Go loops for every scale, including subnormal, inf and NaN scales.
template <int QT, int ORDER, bool VEC>
__global__ void __launch_bounds__(256) dequantize_kernel(const uint8_t *__restrict__ blocks, int64_t nblocks,
                                                       float *__restrict__ y) {
    const int64_t total = nblocks * 8;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t blk = idx >> 3;
        const int p = (int)(idx & 7);
        float v[4];
        if (QT == CQ_Q4_0) {
            const uint8_t *b = blocks + blk * kQ4Bytes;
            const float d = fp16_bits_to_f32(ld_u16(b));
            int q[4];
            if (ORDER == CQ_ORDER_GO_INTERLEAVED) {
                const uint32_t two = ld_u16(b + 2 + 2 * p);  // bytes 2p, 2p+1 -> values 4p..4p+3
                q[0] = two & 0xF, q[1] = (two >> 4) & 0xF, q[2] = (two >> 8) & 0xF, q[3] = (two >> 12) & 0xF;
            } else {
                const uint8_t *qs = b + 2 + 4 * (p & 3);  // values 4p..4p+3 = low (p<4) or high nibbles
                const uint32_t four = ld_u16(qs) | (ld_u16(qs + 2) << 16);
                const int sh = (p >= 4) ? 4 : 0;
                q[0] = (four >> sh) & 0xF, q[1] = (four >> (8 + sh)) & 0xF, q[2] = (four >> (16 + sh)) & 0xF,
                q[3] = (four >> (24 + sh)) & 0xF;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = mul_like_cpu(d, (float)(q[i] - 8));
        } else {
            const uint8_t *b = blocks + blk * kQ8Bytes;
            const float d = fp16_bits_to_f32(ld_u16(b));
            const uint8_t *qs = b + 2 + 4 * p;
            const uint32_t four = ld_u16(qs) | (ld_u16(qs + 2) << 16);
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = mul_like_cpu(d, (float)(int)(signed char)((four >> (8 * i)) & 0xFF));
        }
        if (VEC) {
            reinterpret_cast<float4 *>(y)[idx] = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) y[idx * 4 + i] = v[i];
        }
    }
}

__device__ __forceinline__ void st_u16(uint8_t *p, uint32_t v) { *reinterpret_cast<unsigned short *>(p) = (unsigned short)v; }

template <int QT, int ORDER>
__device__ __forceinline__ void quantize_block(const float (&v)[kQK], uint8_t *b) {
    if (QT == CQ_Q4_0) {
        float amax = 0.0f, mx = 0.0f;
#pragma unroll
        for (int j = 0; j < kQK; ++j)
            if (amax < fabsf(v[j])) {
                amax = fabsf(v[j]);
                mx = v[j];
            }
        const float d = __fdiv_rn(mx, -8.0f);
        const float id = (d != 0.0f) ? __fdiv_rn(1.0f, d) : 0.0f;
        st_u16(b, __half_as_ushort(__float2half_rn(d)));
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
            uint32_t two = 0;
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const int jj = j + t;
                const int i0 = (ORDER == CQ_ORDER_GO_INTERLEAVED) ? 2 * jj : jj;
                const int i1 = (ORDER == CQ_ORDER_GO_INTERLEAVED) ? 2 * jj + 1 : jj + 16;
                int q0 = (int)__fadd_rn(__fmul_rn(v[i0], id), 8.5f);
                int q1 = (int)__fadd_rn(__fmul_rn(v[i1], id), 8.5f);
                q0 = min(15, (int)(signed char)q0);
                q1 = min(15, (int)(signed char)q1);
                two |= (uint32_t)(((q0 & 0xFF) | ((q1 << 4) & 0xFF)) & 0xFF) << (8 * t);
            }
            st_u16(b + 2 + j, two);
        }
    } else {
        float amax = 0.0f;
#pragma unroll
        for (int j = 0; j < kQK; ++j) {
            const float a = fabsf(v[j]);
            amax = amax > a ? amax : a;
        }
        const float d = __fdiv_rn(amax, 127.0f);
        const float id = (d != 0.0f) ? __fdiv_rn(1.0f, d) : 0.0f;
        st_u16(b, __half_as_ushort(__float2half_rn(d)));
#pragma unroll
        for (int j = 0; j < kQK; j += 2) {
            const int q0 = (int)roundf(__fmul_rn(v[j], id));
            const int q1 = (int)roundf(__fmul_rn(v[j + 1], id));
            st_u16(b + 2 + j, (uint32_t)(q0 & 0xFF) | ((uint32_t)(q1 & 0xFF) << 8));
        }
    }
}

// One thread quantizes one block of 32 values, sequentially, so that "first element with
// the largest magnitude" and every rounding follow the reference shaders literally:
// tensor/internal/metal/kernels/quantized.metal:4187-4211 (Q4_0), :4129-4145 (Q8_0).
// Multiplies and adds are issued with explicit rounding intrinsics so the compiler cannot
// contract v*id + 8.5 into one fused operation.
// Bound: HBM (4 bytes in, 0.56 / 1.06 out per value).  A thread that fetched its own 128 bytes touched 32 lines per
// load instruction and wrote its block two bytes at a time; now the CTA's 128 blocks pass through shared memory in both
// directions, so global accesses are whole lines.  Rows of 36 words keep the 16-byte accesses of both sides free of
// bank conflicts (8 lanes x 4 words cover the 32 banks).  11008 x 4096 Q4_0, quantize and dequantize: 90.0 -> 70.7 us.
constexpr int kQuantThreads = 128, kQuantPitch = 36;
template <int QT, int ORDER>
__global__ void __launch_bounds__(kQuantThreads) quantize_rows_kernel(const float *__restrict__ w, int64_t nblocks,
                                                                    uint8_t *__restrict__ blocks) {
    constexpr int BB = QT == CQ_Q4_0 ? kQ4Bytes : kQ8Bytes;
    __shared__ __align__(16) float in[kQuantThreads * kQuantPitch];
    __shared__ __align__(16) uint8_t out[kQuantThreads * BB];
    const int64_t blk0 = (int64_t)blockIdx.x * kQuantThreads;
    const int count = (int)(nblocks - blk0 < kQuantThreads ? nblocks - blk0 : kQuantThreads);  // blocks of this CTA
    const float *src = w + blk0 * kQK;
    if ((reinterpret_cast<uintptr_t>(w) & 15) == 0) {
        float4 t[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int f = threadIdx.x + i * kQuantThreads;  // 16-byte pieces, eight per block
            if (f < 8 * count) t[i] = reinterpret_cast<const float4 *>(src)[f];
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int f = threadIdx.x + i * kQuantThreads;
            if (f < 8 * count) *reinterpret_cast<float4 *>(&in[(f >> 3) * kQuantPitch + 4 * (f & 7)]) = t[i];
        }
    } else {
        for (int f = threadIdx.x; f < kQK * count; f += kQuantThreads) in[(f >> 5) * kQuantPitch + (f & 31)] = src[f];
    }
    __syncthreads();
    float v[kQK];
    if ((int)threadIdx.x < count) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float4 t = *reinterpret_cast<const float4 *>(&in[threadIdx.x * kQuantPitch + 4 * i]);
            v[4 * i] = t.x, v[4 * i + 1] = t.y, v[4 * i + 2] = t.z, v[4 * i + 3] = t.w;
        }
        quantize_block<QT, ORDER>(v, out + threadIdx.x * BB);
    }
    __syncthreads();
    uint8_t *dst = blocks + blk0 * BB;  // blk0 * BB is a multiple of 16
    const int bytes = count * BB;
    if ((reinterpret_cast<uintptr_t>(blocks) & 15) == 0) {
        for (int i = threadIdx.x; i < bytes / 16; i += kQuantThreads) reinterpret_cast<uint4 *>(dst)[i] = reinterpret_cast<const uint4 *>(out)[i];
        for (int i = (bytes & ~15) + 2 * threadIdx.x; i < bytes; i += 2 * kQuantThreads) st_u16(dst + i, ld_u16(out + i));
    } else {
        for (int i = 2 * threadIdx.x; i < bytes; i += 2 * kQuantThreads) st_u16(dst + i, ld_u16(out + i));
    }
}
// One warp per block of 32 activations, as tensor/internal/cuda/kernels/quantized.cu:
// 3521-3558: xor-butterfly max and sum, d = amax/127, q = roundf(x/d) by true division.
__global__ void __launch_bounds__(256) quantize_q8_1_kernel(const float *__restrict__ x, int64_t m, int64_t k, int64_t ldx,
                                                          uint8_t *__restrict__ out) {
    const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= m * k) return;  // m*k is a multiple of 32: whole warps leave together
    const int64_t row = gid / k, col = gid - row * k;
    const float xi = x[row * ldx + col];
    float amax = fabsf(xi), sum = xi;
#pragma unroll
    for (int mask = 16; mask > 0; mask >>= 1) {
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, mask, 32));
        sum += __shfl_xor_sync(0xffffffffu, sum, mask, 32);
    }
    const float d = __fdiv_rn(amax, 127.0f);
    const int q = (amax == 0.0f) ? 0 : (int)roundf(__fdiv_rn(xi, d));
    uint8_t *b = out + (gid >> 5) * kQ81Bytes;
    const int lane = threadIdx.x & 31;
    b[4 + lane] = (uint8_t)(q & 0xFF);
    if (lane == 0) {
        st_u16(b, __half_as_ushort(__float2half_rn(d)));
        st_u16(b + 2, __half_as_ushort(__float2half_rn(sum)));
    }
}

// Rows of blocks and rows of x copied with their length rounded up: zero blocks and zero values follow the last ones.
// A warp per row, 16 bytes per lane and trip: source rows start at any even address, so a lane reads the five aligned words
// around its 16 bytes and shifts them into place.  A word that only touches a row's end lies within four bytes that hold a byte of the row.
constexpr int kPadWarps = 8;
__global__ void __launch_bounds__(32 * kPadWarps) pad_rows_kernel(const uint8_t *__restrict__ w, int64_t n, int row_bytes, int row_out,
                                                                uint8_t *__restrict__ w_out, const float *__restrict__ x, int64_t m, int k, int64_t ldx,
                                                                float *__restrict__ x_out, int k_out) {
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * kPadWarps + (threadIdx.x >> 5);
    if (row < n) {
        const uint8_t *src = w + row * row_bytes;
        const uint32_t odd = (uint32_t)(reinterpret_cast<uintptr_t>(src) & 2);
        const uint8_t *base = src - odd;
        uint4 *dst = reinterpret_cast<uint4 *>(w_out + row * row_out);
#pragma unroll 4
        for (int c = lane; c < row_out / 16; c += 32) {
            uint32_t v[5], o[4];
#pragma unroll
            for (int i = 0; i < 5; ++i) {
                const int at = 16 * c + 4 * i;  // this word holds bytes at - odd .. at - odd + 3 of the row
                v[i] = at - (int)odd < row_bytes && (i < 4 || odd) ? __ldg(reinterpret_cast<const uint32_t *>(base + at)) : 0u;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int at = 16 * c + 4 * i;
                o[i] = __funnelshift_r(v[i], v[i + 1], 8 * odd);
                if (at + 4 > row_bytes) o[i] = at + 2 == row_bytes ? o[i] & 0xFFFFu : (at >= row_bytes ? 0u : o[i]);
            }
            dst[c] = make_uint4(o[0], o[1], o[2], o[3]);
        }
    } else if (row < n + m) {
        const float *src = x + (row - n) * ldx;
        float *dst = x_out + (row - n) * k_out;
        for (int i = lane; i < k_out; i += 32) dst[i] = i < k ? src[i] : 0.0f;
    }
}

}  // namespace

cq_status launch_pad_rows(cq_ctx *ctx, int qtype, const void *w, int64_t n, void *w_out, const float *x, int64_t m, int64_t k, int64_t ldx, float *x_out,
                          int64_t k_out) {
    const int bb = qtype == CQ_Q4_0 ? kQ4Bytes : kQ8Bytes;
    pad_rows_kernel<<<(unsigned)((n + m + kPadWarps - 1) / kPadWarps), 32 * kPadWarps, 0, ctx->stream>>>(
        static_cast<const uint8_t *>(w), n, (int)(k / kQK) * bb, (int)(k_out / kQK) * bb, static_cast<uint8_t *>(w_out), x, m, (int)k, ldx, x_out, (int)k_out);
    CQ_CUDA(ctx, cudaGetLastError());
    return CQ_OK;
}

cq_status launch_dequantize(cq_ctx *ctx, int qtype, int order, const void *blocks, int64_t nblocks, float *y) {
    const bool vec = (reinterpret_cast<uintptr_t>(y) & 15) == 0;
    if ((reinterpret_cast<uintptr_t>(blocks) & 1) != 0) return cq_fail(ctx, CQ_ERR_INVALID_ARG, "blocks must be 2-byte aligned");
    const int64_t total = nblocks * 8;
    const int threads = 256;
    int64_t grid64 = (total + threads - 1) / threads;
    const int64_t cap = (int64_t)ctx->sm_count * 64;
    const unsigned grid = (unsigned)(grid64 < cap ? grid64 : cap);
    const uint8_t *b = static_cast<const uint8_t *>(blocks);
#define CQ_DQ(QT, ORD)                                                                                  \
    do {                                                                                                \
        if (vec) dequantize_kernel<QT, ORD, true><<<grid, threads, 0, ctx->stream>>>(b, nblocks, y);    \
        else dequantize_kernel<QT, ORD, false><<<grid, threads, 0, ctx->stream>>>(b, nblocks, y);       \
    } while (0)
    if (qtype == CQ_Q4_0 && order == CQ_ORDER_GO_INTERLEAVED) CQ_DQ(CQ_Q4_0, 0);
    else if (qtype == CQ_Q4_0) CQ_DQ(CQ_Q4_0, 1);
    else CQ_DQ(CQ_Q8_0, 0);
#undef CQ_DQ
    CQ_CUDA(ctx, cudaGetLastError());
    return CQ_OK;
}

cq_status launch_quantize_rows(cq_ctx *ctx, int qtype, int order, const float *w, int64_t nblocks, void *blocks) {
    if ((reinterpret_cast<uintptr_t>(blocks) & 1) != 0) return cq_fail(ctx, CQ_ERR_INVALID_ARG, "blocks must be 2-byte aligned");
    if ((reinterpret_cast<uintptr_t>(w) & 3) != 0) return cq_fail(ctx, CQ_ERR_INVALID_ARG, "w must be 4-byte aligned");
    const int threads = kQuantThreads;
    const unsigned grid = (unsigned)((nblocks + threads - 1) / threads);
    uint8_t *b = static_cast<uint8_t *>(blocks);
    if (qtype == CQ_Q4_0 && order == CQ_ORDER_GO_INTERLEAVED)
        quantize_rows_kernel<CQ_Q4_0, 0><<<grid, threads, 0, ctx->stream>>>(w, nblocks, b);
    else if (qtype == CQ_Q4_0)
        quantize_rows_kernel<CQ_Q4_0, 1><<<grid, threads, 0, ctx->stream>>>(w, nblocks, b);
    else
        quantize_rows_kernel<CQ_Q8_0, 0><<<grid, threads, 0, ctx->stream>>>(w, nblocks, b);
    CQ_CUDA(ctx, cudaGetLastError());
    return CQ_OK;
}

cq_status launch_quantize_q8_1(cq_ctx *ctx, const float *x, int64_t m, int64_t k, int64_t ldx, void *out) {
    if ((reinterpret_cast<uintptr_t>(out) & 1) != 0) return cq_fail(ctx, CQ_ERR_INVALID_ARG, "q8_1 output must be 2-byte aligned");
    const int threads = 256;
    const unsigned grid = (unsigned)((m * k + threads - 1) / threads);
    quantize_q8_1_kernel<<<grid, threads, 0, ctx->stream>>>(x, m, k, ldx, static_cast<uint8_t *>(out));
    CQ_CUDA(ctx, cudaGetLastError());
    return CQ_OK;
}
