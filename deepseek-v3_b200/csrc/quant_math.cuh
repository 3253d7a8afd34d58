// Arithmetic of act_quant shared by the stand-alone kernel and the GEMM kernels that quantise in their prologue.
//
// Bit-exactness contract (what the reference's kernel computes when compiled for a GPU, inference/kernel.py:23-35):
//   amax = max|x| (NaN operands dropped) ; amax = max(amax, 1e-4f)
//   s = div.full.f32(amax, 448) ; [ue8m0: s = exp2(ceil(log2(s)))]
//   y = cvt.rn.satfinite.e4m3(div.full.f32(x, s))
// For the fp32 scale format the quotient is formed as x * rcp.approx.f32(s): on sm_100 this is
// bit-identical to div.full.f32(x, s) for every bf16 x and every scale a bf16 block maximum can
// produce (checked exhaustively on a B200: 5.3e8 (amax, x) pairs, no mismatch), and it needs one
// reciprocal per block instead of one division per element.
#pragma once

#include "common.cuh"

namespace dsv3 {

__device__ __forceinline__ float scale_from_amax(float amax, int scale_fmt) {
    amax = fmaxf(amax, 1e-4f);
    float s = div_full(amax, 448.0f);
    if (scale_fmt == DSV3_SCALE_FMT_UE8M0) s = exp2f(ceilf(log2f(s)));
    return s;
}

__device__ __forceinline__ float amax8(const uint4& v) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    float m = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m = fmaxf(m, fabsf(bf16_bits_to_float(w[i] & 0xFFFFu)));
        m = fmaxf(m, fabsf(__uint_as_float(w[i] & 0xFFFF0000u)));
    }
    return m;
}

__device__ __forceinline__ float rcp_approx(float s) {
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(s));
    return r;
}

// kRcp: quotient as x * rcp.approx(s) (fp32 scale format) instead of div.full(x, s).
template <bool kRcp>
__device__ __forceinline__ uint2 quant8(const uint4& v, float s) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint16_t p[4];
    const float r = kRcp ? rcp_approx(s) : 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float xl = bf16_bits_to_float(w[i] & 0xFFFFu), xh = __uint_as_float(w[i] & 0xFFFF0000u);
        const float lo = kRcp ? __fmul_rn(xl, r) : div_full(xl, s);
        const float hi = kRcp ? __fmul_rn(xh, r) : div_full(xh, s);
        p[i] = cvt_e4m3x2(lo, hi);
    }
    return make_uint2(static_cast<uint32_t>(p[0]) | (static_cast<uint32_t>(p[1]) << 16),
                      static_cast<uint32_t>(p[2]) | (static_cast<uint32_t>(p[3]) << 16));
}

// silu(a) = a / (1 + exp(-a)) evaluated in fp32 and rounded to bf16: the value of the framework's bf16 kernel, which
// evaluates it with expf and an IEEE division.
static __device__ __noinline__ float silu_exact(float a) {
    return __bfloat162float(__float2bfloat16_rn(a / (1.0f + expf(-a))));
}

__device__ __forceinline__ uint32_t swiglu2_exact(uint32_t a2, uint32_t b2) {
    const float lo = silu_exact(bf16_bits_to_float(a2 & 0xFFFFu)), hi = silu_exact(__uint_as_float(a2 & 0xFFFF0000u));
    return pack_bf16x2(lo * bf16_bits_to_float(b2 & 0xFFFFu), hi * __uint_as_float(b2 & 0xFFFF0000u));
}

// h = bf16(bf16(silu(a)) * b) for eight bf16 pairs.
// The fast form a * rcp(1 + ex2(-a log2 e)) is within 2^-19.5 of the exact form for |a| <= 15 (ex2: 2 ulp, its rounded
// argument 1.2 |a| ulp, rcp 1 ulp, two roundings, and 2 ulp for the exact form's own expf).  It is rounded to bf16 once a
// little below and once a little above itself: where the two agree they are the exact form's value, where they
// disagree (0.05 % of values) or a value lies outside that range the exact form is evaluated.  16 instructions per
// value instead of 40; the exact form is a call, since inlined into an unrolled epilogue it outgrew the instruction cache
// (20000 cycles per tile).
__device__ __forceinline__ uint4 swiglu8(const uint4& a, const uint4& b) {
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
    constexpr float kLog2e = 1.44269504088896340736f;
    constexpr float kEps = 1.34e-6f;       // 2^-19.5
    uint32_t h[4], diff[4];
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
        const float2 lo2 = __fmul2_rn(s2, make_float2(1.0f - kEps, 1.0f - kEps)), hi2 = __fmul2_rn(s2, make_float2(1.0f + kEps, 1.0f + kEps));
        const uint32_t below = pack_bf16x2(lo2.x, lo2.y);
        const uint32_t above = pack_bf16x2(hi2.x, hi2.y);
        diff[i] = below ^ above;
        top = __hmax2_nan(top, __habs2(*reinterpret_cast<const __nv_bfloat162*>(&aw[i])));
        const float2 h2 = __fmul2_rn(make_float2(bf16_bits_to_float(above & 0xFFFFu), __uint_as_float(above & 0xFFFF0000u)),
                                     make_float2(bf16_bits_to_float(bw[i] & 0xFFFFu), __uint_as_float(bw[i] & 0xFFFF0000u)));
        h[i] = pack_bf16x2(h2.x, h2.y);
    }
    const bool far = !__hble2(top, __float2bfloat162_rn(15.0f));
    if (far || (diff[0] | diff[1] | diff[2] | diff[3]) != 0u) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (far || diff[i] != 0u) h[i] = swiglu2_exact(aw[i], bw[i]);
    }
    return make_uint4(h[0], h[1], h[2], h[3]);
}

}  // namespace dsv3
