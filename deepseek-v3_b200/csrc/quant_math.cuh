// Arithmetic of act_quant shared by the stand-alone kernel and the GEMM kernels that quantise in their prologue.
//
// Bit-exactness contract (what the reference's kernel computes when compiled for a GPU, inference/kernel.py:23-35):
//   amax = max|x| (NaN operands dropped) ; amax = max(amax, 1e-4f)
//   s = div.full.f32(amax, 448) ; [ue8m0: s = exp2(ceil(log2(s)))]
//   y = cvt.rn.satfinite.e4m3(div.full.f32(x, s))
// The quotient is formed as x * rcp.approx.f32(s), one reciprocal per block instead of one division per element.  For the fp32
// scale format this is bit-identical to div.full.f32(x, s) on sm_100 for every bf16 x and every scale a bf16 block maximum
// can produce (checked exhaustively on a B200: 5.3e8 (amax, x) pairs, no mismatch).  For ue8m0 both are exact: a scale is a power of
// two from 2^-22 to 2^120, whose reciprocal rcp.approx gives exactly (every one of them checked on a B200), or infinite.
#pragma once

#include "common.cuh"

namespace dsv3 {

__device__ __forceinline__ float scale_from_amax(float amax, int scale_fmt) {
    amax = fmaxf(amax, 1e-4f);
    float s = div_full(amax, 448.0f);
    if (scale_fmt == DSV3_SCALE_FMT_UE8M0) s = exp2f(ceilf(log2f(s)));
    return s;
}

__device__ __forceinline__ uint32_t max_bf16x2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("max.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}

// max|x| of eight bf16 values
__device__ __forceinline__ float amax8(const uint4& v) {
    // two values to a word; a NaN gives way to the other operand, and a lane of nothing but NaN returns one, which fmaxf drops
    const uint32_t m = max_bf16x2(max_bf16x2(v.x & 0x7FFF7FFFu, v.y & 0x7FFF7FFFu), max_bf16x2(v.z & 0x7FFF7FFFu, v.w & 0x7FFF7FFFu));
    return fmaxf(__uint_as_float(m << 16), __uint_as_float(m & 0xFFFF0000u));
}

__device__ __forceinline__ float rcp_approx(float s) {
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(s));
    return r;
}

// The scales of a half-warp's kU blocks, whose values lie eight to a lane (m: a lane's maxima).  The lanes share the work out: in the
// first exchanges each gives away the blocks that it will not finish, so that a lane ends up with one block's maximum (five
// exchanges for four blocks instead of sixteen) and forms one scale and one reciprocal instead of four (for ue8m0 a logarithm and an
// exponential each): with a block at a time the passes that are not at the HBM rate were bound by instructions.  B200, us, a block at
// a time and, for ue8m0, divisions / so: 512 x 7168 3.20 / 2.72, ue8m0 4.36 / 2.84; 1003 x 7168 3.48 / 3.10, 4.70 / 3.25; 4096 x 2048 4.07 / 3.61, 5.31 /
// 3.77; 16384 x 7168 52.9 / 52.8, 58.4 / 52.8; swiglu_quant 8192 x 18432 133.5 / 126.9, 153.5 / 132.7.  (Where a CTA quantises a few blocks
// for itself, under the loads of its weights, the exchanges only lengthen the chain: 7168 -> 1536 at one row 5.97 / 6.29; the
// dispatch of the expert layer, whose rounds of blocks are few, 64 experts and 2048 tokens 12.9 / 13.6.)  Returns the scale of block own_block<kU>(), which the quarter (kU = 4) or half of the lanes hold; r: every
// block's reciprocal, in all lanes.  All 32 lanes take part.
template <int kU>
__device__ __forceinline__ int own_block() {
    const int lane = threadIdx.x & 31;
    return kU == 4 ? (lane >> 2) & 3 : (kU == 2 ? (lane >> 3) & 1 : 0);
}
template <int kU>
__device__ __forceinline__ bool own_block_writer() { return (threadIdx.x & (16 / kU - 1)) == 0; }
template <int kU>
__device__ __forceinline__ float block_scales(const float (&m)[kU], int scale_fmt, float (&r)[kU]) {
    static_assert(kU == 1 || kU == 2 || kU == 4, "blocks of a half-warp");
    const int lane = threadIdx.x & 31;
    float keep;
    if constexpr (kU == 4) {
        const bool hi = lane & 8;
        const float a = fmaxf(hi ? m[2] : m[0], __shfl_xor_sync(0xffffffffu, hi ? m[0] : m[2], 8));
        const float b = fmaxf(hi ? m[3] : m[1], __shfl_xor_sync(0xffffffffu, hi ? m[1] : m[3], 8));
        const bool odd = lane & 4;
        keep = fmaxf(odd ? b : a, __shfl_xor_sync(0xffffffffu, odd ? a : b, 4));
    } else if constexpr (kU == 2) {
        const bool hi = lane & 8;
        keep = fmaxf(hi ? m[1] : m[0], __shfl_xor_sync(0xffffffffu, hi ? m[0] : m[1], 8));
        keep = fmaxf(keep, __shfl_xor_sync(0xffffffffu, keep, 4));
    } else {
        keep = fmaxf(m[0], __shfl_xor_sync(0xffffffffu, m[0], 8));
        keep = fmaxf(keep, __shfl_xor_sync(0xffffffffu, keep, 4));
    }
    keep = fmaxf(keep, __shfl_xor_sync(0xffffffffu, keep, 2));
    keep = fmaxf(keep, __shfl_xor_sync(0xffffffffu, keep, 1));
    const float s = scale_from_amax(keep, scale_fmt);
    const float mine = rcp_approx(s);
#pragma unroll
    for (int u = 0; u < kU; ++u) r[u] = kU == 1 ? mine : __shfl_sync(0xffffffffu, mine, (lane & 16) | (u * (16 / kU)));
    return s;
}

// Eight values times the reciprocal of their block's scale.
__device__ __forceinline__ uint2 quant8(const uint4& v, float r) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint16_t p[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 q = __fmul2_rn(make_float2(bf16_bits_to_float(w[i] & 0xFFFFu), __uint_as_float(w[i] & 0xFFFF0000u)), make_float2(r, r));
        p[i] = cvt_e4m3x2(q.x, q.y);
    }
    return make_uint2(static_cast<uint32_t>(p[0]) | (static_cast<uint32_t>(p[1]) << 16),
                      static_cast<uint32_t>(p[2]) | (static_cast<uint32_t>(p[3]) << 16));
}

// silu(a) = a / (1 + exp(-a)) evaluated in fp32 and rounded to bf16: the value of the framework's bf16 kernel, which
// evaluates it with expf and an IEEE division.
static __device__ __noinline__ float silu_exact(float a) {
    return __bfloat162float(__float2bfloat16_rn(a / (1.0f + expf(-a))));
}

// h = bf16(bf16(silu(a)) * b) for eight bf16 pairs.
// silu's fast form, a * rcp(1 + ex2(-a log2 e)), is within 13 ulp of fp32 of the exact one, and rounds to the same bf16 value for every
// bf16 a but -87.5, -88 and -88.5, whose reciprocals are flushed (all 65536 checked on a B200): those are a * exp(a / 2) * exp(a / 2).
// The product of two bf16 values, rounded once, is what it is by way of fp32: of its at most 16 bits fp32 drops one only below 2^-134, where either
// way ends at zero.
// The exact form by a call where the fast one lay near a rounding boundary (0.05 % of values, 13 % of a warp's trips) cost the epilogue of a
// 128-token tile 2300 of 9700 cycles, the check, the separate product and the maximum per word another 600.  us, with them / without: w1 and w3 of 64
// experts of 2048 x 1408, 512 rows each 256 / 225, of 32 of 7168 x 2048 485 / 451; swiglu_quant 8192 x 18432 127 / 111, ue8m0 138 / 112,
// 2048 x 2048 6.8 / 5.0; MLP 2048 -> 2816 at 500 rows 28.1 / 26.6.
__device__ __forceinline__ uint4 swiglu8(const uint4& a, const uint4& b) {
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
    constexpr float kLog2e = 1.44269504088896340736f;
    uint32_t h[4];
    __nv_bfloat162 top = __float2bfloat162_rn(0.0f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        // two values to an FP32 instruction: with one each, swiglu_quant was bound by issue (8192 x 18432 142.9 us, 134.0 so)
        const float2 a2 = make_float2(bf16_bits_to_float(aw[i] & 0xFFFFu), __uint_as_float(aw[i] & 0xFFFF0000u));
        const float2 x2 = __fmul2_rn(a2, make_float2(-kLog2e, -kLog2e));
        float2 e2, r2;
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e2.x) : "f"(x2.x));
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e2.y) : "f"(x2.y));
        e2 = __fadd2_rn(e2, make_float2(1.0f, 1.0f));
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r2.x) : "f"(e2.x));
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r2.y) : "f"(e2.y));
        const float2 s2 = __fmul2_rn(a2, r2);
        const __nv_bfloat162 silu = __floats2bfloat162_rn(s2.x, s2.y), h2 = __hmul2(silu, *reinterpret_cast<const __nv_bfloat162*>(&bw[i]));
        h[i] = *reinterpret_cast<const uint32_t*>(&h2);
        top = __hmax2_nan(top, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&aw[i])));
    }
    if (!__hble2(top, __float2bfloat162_rn(87.0f))) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int up = i & 1 ? 0 : 16;              // shifts the value to the upper half of the word
            const float v = __uint_as_float((aw[i / 2] << up) & 0xFFFF0000u), w = __uint_as_float((bw[i / 2] << up) & 0xFFFF0000u);
            if (v > -88.7f && v < -87.0f) {
                float root;
                asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(root) : "f"(v * (0.5f * kLog2e)));
                const uint32_t r = __bfloat16_as_ushort(__float2bfloat16_rn(__bfloat162float(__float2bfloat16_rn(v * root * root)) * w));
                h[i / 2] = up ? (h[i / 2] & 0xFFFF0000u) | r : (h[i / 2] & 0xFFFFu) | (r << 16);
            }
        }
    }
    return make_uint4(h[0], h[1], h[2], h[3]);
}

}  // namespace dsv3
