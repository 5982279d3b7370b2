// What the GEMMs share that dequantize raw blocks into tensor memory (gemm_pair_tmem.cu: CQ_ACT_F32 and
// CQ_ACT_F16, on CTA pairs; gemm_blocks.cu: CQ_ACT_Q8_1): shares of the work, the sum of partial tiles, tensor maps and launches.
#pragma once
#include "common.cuh"
#include "tcgen05.cuh"

namespace {

constexpr int GP_ROWS = 128;    // weight rows per CTA
constexpr int GP_CHUNK = 256;   // values of k per work item and raw stage

struct GpParams {
    float *y;
    int64_t ldy;
    float *part;           // [2 * shares][NB][TILE]: a share's first tile, and its last
    const float *xscale;   // of activations as hi + lo: 2^-e of each batch row, negative for rows to be computed in plain f32
    const float *x;        // the operands as given, for what is computed in plain f32
    const uint8_t *w;
    const float *bias;     // [n] or null
    int64_t ldx;
    int m, n, k, order;
    int mtiles, nchunks, total, per_share;
    int *err;
};

// y of the tiles (TILE weight rows x NB batch rows) whose k range several shares hold: their partial tiles, added in order.
// Block = (tile, 1024 / TILE batch rows).
template <int TILE, int NB>
__global__ void __launch_bounds__(256) gp_sum_kernel(const GpParams p) {
    pdl_launch_dependents();
    pdl_wait_prior();
    constexpr int PER = TILE / 4;  // threads per batch row
    const int t = blockIdx.x, lc = blockIdx.y * (256 / PER) + threadIdx.x / PER;
    const int group = t / p.mtiles, col = (t - group * p.mtiles) * NB + lc;
    const int first = (t * p.nchunks) / p.per_share, last = ((t + 1) * p.nchunks - 1) / p.per_share;
    if (first == last || col >= p.m) return;  // one share had the whole k range and wrote y itself
    const int r = (threadIdx.x % PER) * 4;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    const bool ends = (first * p.per_share) / p.nchunks != t;  // the first share had an earlier tile too: this one is its second slot
    for (int c = first; c <= last; c += 4) {
        // Four partial tiles in flight, and none twice.  (us of the call with one at a time / four / eight / eight whose loads past the
        // last repeat it: f16 128 x 4096 x 4096 15.4 / 14.6 / 14.4 / 15.7, 128 x 11008 x 4096 22.6 / 22.2 / 22.8 / 22.7; f32 512 x 11008 x
        // 4096 112.4 / 112.8 / 114.1 / 114.6; Q8_1 64 x 700 x 14336, 19 of them, 21.9 / 20.9 / 20.5 / 20.9.)
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (c + u <= last) v[u] = *reinterpret_cast<const float4 *>(p.part + ((int64_t)(2 * (c + u) + (c + u == first && ends ? 1 : 0)) * NB + lc) * TILE + r);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (c + u <= last) acc.x += v[u].x, acc.y += v[u].y, acc.z += v[u].z, acc.w += v[u].w;
    }
    const int64_t j = (int64_t)group * TILE + r;
    if (p.bias) {
        if (j < p.n) acc.x += p.bias[j];
        if (j + 1 < p.n) acc.y += p.bias[j + 1];
        if (j + 2 < p.n) acc.z += p.bias[j + 2];
        if (j + 3 < p.n) acc.w += p.bias[j + 3];
    }
    float *dst = p.y + (int64_t)col * p.ldy + j;
    if (j + 3 < p.n && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
        *reinterpret_cast<float4 *>(dst) = acc;
    } else {
        if (j < p.n) dst[0] = acc.x;
        if (j + 1 < p.n) dst[1] = acc.y;
        if (j + 2 < p.n) dst[2] = acc.z;
        if (j + 3 < p.n) dst[3] = acc.w;
    }
}

// Eight nibbles -> four pairs (v0,v4)(v1,v5)(v2,v6)(v3,v7) of -8 .. 7: 1024 + q assembled by one mask-or, 1032 taken off exactly.
__device__ __forceinline__ void gp_numbers_q4(uint32_t n, __half2 (&q)[4]) {
    const __half2 k1032 = __halves2half2(__ushort_as_half(0x6408), __ushort_as_half(0x6408));
    const __half2 k16th = __halves2half2(__ushort_as_half(0x2C00), __ushort_as_half(0x2C00));
    const __half2 km72 = __halves2half2(__ushort_as_half(0xD480), __ushort_as_half(0xD480));
    const uint32_t n8 = n >> 8;
    uint32_t t0 = (n & 0x000F000Fu) | 0x64006400u, t1 = (n & 0x00F000F0u) | 0x64006400u;
    uint32_t t2 = (n8 & 0x000F000Fu) | 0x64006400u, t3 = (n8 & 0x00F000F0u) | 0x64006400u;
    q[0] = __hsub2(*reinterpret_cast<__half2 *>(&t0), k1032);
    q[1] = __hfma2(*reinterpret_cast<__half2 *>(&t1), k16th, km72);
    q[2] = __hsub2(*reinterpret_cast<__half2 *>(&t2), k1032);
    q[3] = __hfma2(*reinterpret_cast<__half2 *>(&t3), k16th, km72);
}
// Four int8 -> two pairs, natural order.
__device__ __forceinline__ void gp_numbers_q8(uint32_t n, __half2 (&q)[2]) {
    const __half2 k1152 = __halves2half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480));
    const uint32_t u = n ^ 0x80808080u;
    uint32_t t0 = __byte_perm(u, 0x64646464u, 0x4140), t1 = __byte_perm(u, 0x64646464u, 0x4342);
    q[0] = __hsub2(*reinterpret_cast<__half2 *>(&t0), k1152);
    q[1] = __hsub2(*reinterpret_cast<__half2 *>(&t1), k1152);
}

// Raw blocks as a 2-D tensor of 2-byte elements, box = 256 values of k x 128 rows.
bool gp_w_map(CUtensorMap *map, const void *w, int64_t n, int64_t row_bytes, int row_chunk) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)(row_bytes / 2), (cuuint64_t)n};
    cuuint64_t strides[1] = {(cuuint64_t)row_bytes};
    cuuint32_t box[2] = {(cuuint32_t)(row_chunk / 2), (cuuint32_t)GP_ROWS};
    cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void *>(w), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// Activations as [hi / lo][k / 64][m][64]: ONE copy then brings a whole stage (`slabs` times 64 k of `rows` batch rows, both
// halves of a split) as the 64-wide swizzled boxes the MMA reads; one thread starts a copy only every few hundred cycles.
bool gp_x_map(CUtensorMap *map, const void *x16, int64_t m, int64_t k, size_t lo_offset, int rows, int slabs) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    const int parts = lo_offset ? 2 : 1;
    cuuint64_t dims[4] = {64u, (cuuint64_t)m, (cuuint64_t)(k / 64), (cuuint64_t)parts};
    cuuint64_t strides[3] = {(cuuint64_t)k * 2, 128u, lo_offset ? (cuuint64_t)lo_offset : (cuuint64_t)k * 2};
    cuuint32_t box[4] = {64u, (cuuint32_t)rows, (cuuint32_t)slabs, (cuuint32_t)parts};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void *>(x16), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <typename Kern, typename... Args>
cq_status gp_launch(cq_ctx *ctx, Kern kern, dim3 grid, int block, size_t smem, bool cluster, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (ctx->tune.pdl) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = 2, attr[na].val.clusterDim.y = 1, attr[na++].val.clusterDim.z = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    CQ_CUDA(ctx, cudaLaunchKernelEx(&cfg, kern, args...));
    return CQ_OK;
}


// How a call's (tile, chunk) items are shared out among at most `max_shares` CTAs or pairs of them, and what of scratch that
// takes behind its operands.  A call that is being captured with room for the operands but not for partial tiles gives whole
// tiles to the shares, which need none.
struct GpShares {
    int64_t tiles = 0;
    unsigned shares = 0;
    bool cut = false;   // some tile's k range lies in several shares: gp_sum_kernel
    size_t part_bytes = 0;
};
inline cq_status gp_share_out(cq_ctx *ctx, GpParams &p, int tile, int nb, int max_shares, size_t operand_bytes, GpShares &s) {
    p.mtiles = (p.m + nb - 1) / nb;
    p.nchunks = p.k / GP_CHUNK;
    s.tiles = (((int64_t)p.n + tile - 1) / tile) * (int64_t)p.mtiles;
    const int64_t total = s.tiles * p.nchunks;
    if (total > 0x3FFFFFFF / (tile / GP_ROWS)) return cq_fail(ctx, CQ_ERR_TOO_LARGE, "gemm: too many tiles");
    int64_t per = (total + max_shares - 1) / max_shares;
    if (per < 2) per = total < 2 ? total : 2;
    auto part = [&] { return per % p.nchunks != 0 ? (size_t)2 * ((total + per - 1) / per) * nb * tile * 4 : size_t(0); };
    if (operand_bytes + part() > ctx->scratch_bytes && cq_stream_capturing(ctx)) per = (s.tiles + max_shares - 1) / max_shares * p.nchunks;
    s.shares = (unsigned)((total + per - 1) / per);
    s.cut = per % p.nchunks != 0;
    s.part_bytes = part();
    p.total = (int)total, p.per_share = (int)per;
    return CQ_OK;
}

}  // namespace
