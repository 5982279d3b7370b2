// What the two prefill attention kernels share: parameters, exponentials, packing, tensor maps.
#pragma once
#include <cuda_bf16.h>

#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "tcgen05.cuh"

struct FaParams {
    void *o;
    float *lse;             // [b][h][seqlen_q] or null
    int64_t o_batch_stride, o_row_stride, o_head_stride;
    int b, h, h_k, seqlen_q, seqlen_k;
    int causal;
    float scale_log2;       // softmax_scale * log2(e)
    float scale;            // softmax_scale
    int *err;
};

namespace {

constexpr int FA_M = 128;   // query rows per tile
constexpr int FA_N = 128;   // keys per tile


__device__ __forceinline__ void tma_load_3d(uint32_t smem_dst, const CUtensorMap *map, int c0, int c1, int c2, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_dst),
        "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
        : "memory");
}
// kind::f16 instruction descriptor with the operand type: f16 (0) or bf16 (1); D f32; both operands K-major.
__host__ __device__ constexpr uint32_t idesc_16(int mm, int nn, bool bf16) {
    return (1u << 4) | ((bf16 ? 1u : 0u) << 7) | ((bf16 ? 1u : 0u) << 10) | ((uint32_t)(nn >> 3) << 17) | ((uint32_t)(mm >> 4) << 24);
}

// 2^x by the special-function unit (relative error about 2^-22; -inf gives 0)
__device__ __forceinline__ float fast_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

template <bool BF16>
__device__ __forceinline__ uint32_t pack16(float a, float b) {
    if (BF16) {
        const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
        return *reinterpret_cast<const uint32_t *>(&v);
    }
    const __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&v);
}

// Q / K: [b][row][head][d] with strides in elements -> 4-D map (d, head, row, batch); box = 64 x 1 x 128 x 1.
bool make_qk_map(CUtensorMap *map, const void *base, bool bf16, int d, int heads, int rows, int batches, int64_t hs, int64_t rs, int64_t bs) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return false;
    cuuint64_t dims[4] = {(cuuint64_t)d, (cuuint64_t)heads, (cuuint64_t)rows, (cuuint64_t)batches};
    cuuint64_t strides[3] = {(cuuint64_t)hs * 2, (cuuint64_t)rs * 2, (cuuint64_t)bs * 2};
    cuuint32_t box[4] = {64u, 1u, 128u, 1u};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    return fn(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void *>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
}  // namespace

// Two query tiles per CTA (attention_two_tiles.cu); head dimension 64 or 128, V where it lies.
cq_status launch_fmha_two_tiles(cq_ctx *ctx, const CUtensorMap &tq, const CUtensorMap &tk, const CUtensorMap &tv, const FaParams &p, int d, bool bf16);
