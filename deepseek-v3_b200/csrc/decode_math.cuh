// What the two decode-sized kernels (fp8_linear_small.cu, moe_few.cu) do alike: a chunk product of mma.sync on fragments that
// lanes load straight from memory, and the quantisation of a block by a half-warp.
#pragma once

#include "quant_math.cuh"

namespace dsv3 {

constexpr int kChunkK = 128;    // K elements (= bytes) per scale block
constexpr int kRowPad = 64;     // bytes between staged token rows beyond the K range: the 8 lanes of one shared-memory
                                // phase (two token rows x four 16-byte pieces) then hit 8 different bank groups

__device__ __forceinline__ void mma_e4m3(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.f32.e4m3.e4m3.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// 16 weight rows x 8 tokens over one chunk.  Lane 4 g + t holds bytes 16 t .. 16 t + 15 of both 64-byte halves: w of weight rows g
// and g + 8 (half 0: w[0], w[1]; half 1: w[2], w[3]), f0 and f1 of token row g.  The K positions inside a half are permuted
// the same way for both operands.  part[0..1]: weight row g, tokens 2 t and 2 t + 1; part[2..3]: weight row g + 8.
__device__ __forceinline__ void chunk_product(float (&part)[4], const uint4 (&w)[4], const uint4& f0, const uint4& f1) {
    part[0] = part[1] = part[2] = part[3] = 0.0f;
    mma_e4m3(part, w[0].x, w[1].x, w[0].y, w[1].y, f0.x, f0.y);
    mma_e4m3(part, w[0].z, w[1].z, w[0].w, w[1].w, f0.z, f0.w);
    mma_e4m3(part, w[2].x, w[3].x, w[2].y, w[3].y, f1.x, f1.y);
    mma_e4m3(part, w[2].z, w[3].z, w[2].w, w[3].w, f1.z, f1.w);
}

// The scale of a half-warp's block of 128 bf16 values, eight per lane (act_quant's arithmetic).
__device__ __forceinline__ float half_warp_scale(const uint4& v, int scale_fmt) {
    float m = amax8(v);
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 8));
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 4));
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
    return scale_from_amax(m, scale_fmt);
}

}  // namespace dsv3
