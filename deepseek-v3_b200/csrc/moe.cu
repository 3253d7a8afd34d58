// MoE expert loop as grouped GEMMs: C entry points and the combine kernel.
//
// Replaces the Python loop of MoE.forward (inference/model.py:683-689): per local expert i,
//   idx, top = where(indices == i) ; y[idx] += expert(x[idx]) * weights[idx, top, None]
// with bf16 rounding after the product and after every accumulation, in ascending expert order.
#include <type_traits>

#include "gemm_plan.cuh"
#include "quant_math.cuh"

namespace dsv3 {

namespace {

constexpr int kThreads = 256;

// y[t, :] = sum over the token's experts, in ascending expert order, of bf16(o[pos, :] * w), each
// partial sum rounded to bf16 (the arithmetic of `y[idx] += ...` on bf16 tensors); with z, y + z follows (model.py:693).
//   pos [T, topk] int32: row of `o` holding expert output for the j-th smallest expert id of token t, or -1
//   w   [T, topk] bf16 : routing weight of that pair
// Bound by HBM: 2 dim (local pairs + 1 or 2 per token) bytes, and by what a CTA spends besides: its look-up of the token's rows and the
// wait for them behind it, where a rank owns a few of the experts for one or two rows, and two roundings per value.  So the
// arithmetic is packed, two values to an instruction (in fp32 with conversions it bound full rows: 4096 tokens, 128 of 256 experts of
// dim 7168, 89.8 us, so 69.7), and with many tokens a thread takes four 16-byte pieces of a row, two rows at a time: a quarter of the
// CTAs, and eight loads in flight again where both are there (57.4).  us, before / <1, 6> / <4, 2>: 32 of 256 experts of dim 7168,
// 4 tokens 3.3 / 2.8 / 3.8, 333 8.1 / 7.4 / 6.3, 4096 66.0 / 61.1 / 35.8; 128 of them, 333 10.8 / 8.4 / 8.8; 20 of 160 of dim 5120, 333
// 6.1 / 4.7 / 4.8, 4096 43.9 / 32.2 / 20.7; rows of 2048, 64 of 64 experts, make CTAs of 64 threads: 2048 tokens 18.0 / 10.8 / 11.6.  Two
// pieces and four rows lie in between; a list of the rows of several tokens, worked on side by side, did too.
constexpr int kCombineManyTokens = 400, kCombineManyDim = 4096;

// Two bf16 values to a word, each result rounded once to bf16: what a product or sum formed in fp32 and then rounded gives (a
// product of two bf16 values is exact in fp32, or below 2^-134, where either way ends at zero; a sum that is not exact lies too far from a
// tie of bf16 for the first of two roundings to matter).
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t add_bf16x2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("add.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}

template <int kPieces, int kCombineBatch>
__global__ void __launch_bounds__(kThreads, kPieces == 1 ? 5 : 4) moe_combine_kernel(const __nv_bfloat16* __restrict__ o,
                                                                const int* __restrict__ pos,
                                                                const __nv_bfloat16* __restrict__ w,
                                                                const __nv_bfloat16* __restrict__ z,
                                                                __nv_bfloat16* __restrict__ y, int topk, int64_t dim,
                                                                FastDiv ctas_per_row) {
    griddep_launch_dependents();
    griddep_wait();
    const uint32_t t = fast_div(blockIdx.x, ctas_per_row);
    const int* tp = pos + static_cast<int64_t>(t) * topk;
    const unsigned short* tw = reinterpret_cast<const unsigned short*>(w) + static_cast<int64_t>(t) * topk;
    // 8 bf16 = 16 bytes per thread and piece
    const int64_t d = (static_cast<int64_t>(blockIdx.x - t * ctas_per_row.d) * (kPieces * blockDim.x) + threadIdx.x) << 3, step = static_cast<int64_t>(blockDim.x) << 3;
    bool in[kPieces];
    uint4 zv[kPieces];
    uint32_t acc[kPieces][4];
#pragma unroll
    for (int q = 0; q < kPieces; ++q) {
        in[q] = d + q * step < dim;
        zv[q] = z && in[q] ? __ldcs(reinterpret_cast<const uint4*>(z + t * dim + d + q * step)) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[q][e] = 0u;
    }
    for (int j0 = 0; j0 < topk; j0 += kCombineBatch) {
        int r[kCombineBatch];
        uint32_t wf[kCombineBatch];
        uint4 v[kCombineBatch][kPieces];
#pragma unroll
        for (int j = 0; j < kCombineBatch; ++j) {
            r[j] = j0 + j < topk ? __ldg(tp + j0 + j) : -1;
            wf[j] = 0x10001u * __ldg(tw + min(j0 + j, topk - 1));
        }
#pragma unroll
        for (int j = 0; j < kCombineBatch; ++j) {
            if (r[j] < 0) continue;
            const __nv_bfloat16* src = o + static_cast<int64_t>(r[j]) * dim + d;
#pragma unroll
            for (int q = 0; q < kPieces; ++q)
                if (in[q]) v[j][q] = __ldcs(reinterpret_cast<const uint4*>(src + q * step));
        }
#pragma unroll
        for (int j = 0; j < kCombineBatch; ++j) {
            if (r[j] < 0) continue;
#pragma unroll
            for (int q = 0; q < kPieces; ++q) {
                const uint32_t words[4] = {v[j][q].x, v[j][q].y, v[j][q].z, v[j][q].w};
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[q][e] = add_bf16x2(acc[q][e], mul_bf16x2(words[e], wf[j]));
            }
        }
    }
#pragma unroll
    for (int q = 0; q < kPieces; ++q) {
        if (!in[q]) continue;
        if (z) {
            acc[q][0] = add_bf16x2(acc[q][0], zv[q].x);
            acc[q][1] = add_bf16x2(acc[q][1], zv[q].y);
            acc[q][2] = add_bf16x2(acc[q][2], zv[q].z);
            acc[q][3] = add_bf16x2(acc[q][3], zv[q].w);
        }
        *reinterpret_cast<uint4*>(y + t * dim + d + q * step) = make_uint4(acc[q][0], acc[q][1], acc[q][2], acc[q][3]);
    }
}

// Everything in front of the expert GEMMs in one launch: groups the (token, expert) pairs by local expert, orders every
// token's pairs by expert id, quantises every token once (act_quant's arithmetic) and writes its FP8 row to the row of
// each of its local pairs.  Replaces moe_route, act_quant and two gathers (and a conversion of the routing weights).
//
// A CTA owns `tpc` consecutive tokens and needs the rows of their pairs: the first row of every expert (all pairs) plus
// how many pairs of the expert belong to earlier tokens.  Instead of a second launch or a grid barrier every CTA counts
// all pairs itself, 8 bytes per pair from L2 into shared-memory histograms (one CTA doing all the bookkeeping took 59 us
// for 16 K pairs); one large CTA per SM keeps that to 16 pairs per thread.  An expert's rows are in the order of the pairs,
// counted and never drawn from an atomic: where the expert GEMMs cut a tile over K, its place decides the order of its sums,
// so a row's place must not depend on timing.  It also lets several CTAs along y share a CTA's tokens when there are few.
constexpr int kDispMaxExperts = 256;
constexpr int kDispUnroll = 4;
constexpr int kDispThreads = 1024;
constexpr int kDispPairs = kDispThreads;  // own pairs of a CTA: one per thread

struct DispatchParams {
    const uint4* x;                       // bf16 [T, dim]
    const int64_t* indices;               // [T, topk]
    const void* weights;                  // [T, topk], bf16 or fp32
    int weights_bf16;
    int64_t T, P;
    int topk, dim, start, n, tpc, scale_fmt;
    int* seg;                             // [n + 1]
    int* pos_sorted;                      // [T, topk]
    __nv_bfloat16* w_sorted;              // [T, topk]
    uint2* xq;                            // e4m3 [T, dim]
    float* xs;                            // [T, dim / 128]
    uint2* xq_rows;                       // e4m3 [P, dim]
    float* xs_rows;                       // [dim / 128, P]
    int per_y;                            // blocks of a token row that a CTA along y has
    uint32_t by_b[2];                     // 2^32 / that, rounded up; [1]: of the last along y, which may have fewer
    FastDiv div_topk;
};

__global__ void __launch_bounds__(kDispThreads) moe_dispatch_kernel(const DispatchParams p) {
    __shared__ int total[kDispMaxExperts], before[kDispMaxExperts], scan[kDispMaxExperts / 32];
    __shared__ int own_e[kDispPairs], own_row[kDispPairs];
    __shared__ int to_row[kDispPairs], to_rows[kDispPairs];       // a token's local rows, side by side, and how many
    __shared__ __align__(8) uint8_t in_warp[kDispThreads / 32][kDispMaxExperts];      // a warp's own pairs of each expert
    griddep_launch_dependents();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < kDispMaxExperts) {
        total[tid] = 0;
        before[tid] = 0;
    }
    static_assert(sizeof(in_warp) == 8 * kDispThreads, "eight bytes per thread");
    reinterpret_cast<uint2*>(&in_warp[0][0])[tid] = make_uint2(0u, 0u);
    __syncthreads();
    griddep_wait();
    const int topk = p.topk;
    const int64_t t0 = static_cast<int64_t>(blockIdx.x) * p.tpc;
    const int tokens = static_cast<int>(min(static_cast<int64_t>(p.tpc), p.T - t0));
    const int own = tokens * topk;
    const int64_t own0 = t0 * topk;
    const int nb = p.dim / 128;
    const int b_lo = blockIdx.y * p.per_y, b_n = min(p.per_y, nb - b_lo);
    const int items = b_n > 0 ? tokens * b_n : 0;
    // i / b_n is the upper half of i * by_b_n, as long as items * b_n < 2^32 (and b_n > 1)
    const uint32_t by_b_n = p.by_b[b_n == p.per_y ? 0 : 1];
    const bool divide = b_n == 1 || static_cast<uint64_t>(items) * b_n >= (1ull << 32);
    const int lane16 = tid & 15;
    constexpr int kHalfWarps = kDispThreads / 16;
    // With few tokens this kernel is a chain of short steps.  So shared memory is cleared before the wait, the divisions are the host's, and the
    // first round's block, when there is only one round, is on its way while the pairs are counted.  us, one launch behind another, 4, 148 and 600 tokens 3.78 /
    // 3.26, 4.57 / 4.06, 5.79 / 5.29; per layer, 64 experts of
    // 2048 x 1408, 8 of them here, 62 and 300 tokens 37.5 / 36.7, 54.6 / 53.4; a decode layer in a graph, 6 and 16 sequences 70.9 / 70.0, 110.6 / 109.7.
    // (Its own pairs' experts asked for here, too, instead of behind the loop: 0.5 to 1 us slower with 6 and 16; their weights: no change.)
    const bool one_round = items <= kHalfWarps;
    uint4 early = make_uint4(0u, 0u, 0u, 0u);
    if (one_round && (tid >> 4) < items) {
        const int i = tid >> 4, t = b_n == 1 ? i : static_cast<int>(__umulhi(static_cast<uint32_t>(i), by_b_n));
        early = __ldg(p.x + ((t0 + t) * nb + b_lo + (i - t * b_n)) * 16 + lane16);
    }
#pragma unroll 4
    for (int64_t pr = tid; pr < p.P; pr += kDispThreads) {
        const int64_t e = __ldg(p.indices + pr) - p.start;
        if (e >= 0 && e < p.n) atomicAdd(pr < own0 ? &before[e] : &total[e], 1);       // earlier tokens' pairs, and all others
    }
    int mine = -1, rank_in_warp = 0;          // this thread's pair: local expert and its place among the warp's pairs of that expert
    if (warp * 32 < own) {
        if (tid < own) {
            const int64_t e = __ldg(p.indices + own0 + tid);
            own_e[tid] = static_cast<int>(max(min(e, static_cast<int64_t>(0x3fffffff)), static_cast<int64_t>(-1)));
            if (e >= p.start && e - p.start < p.n) mine = static_cast<int>(e - p.start);
        }
        const unsigned same = __match_any_sync(0xffffffffu, mine);
        rank_in_warp = __popc(same & ((1u << lane) - 1u));
        if (mine >= 0 && rank_in_warp == 0) in_warp[warp][mine] = static_cast<uint8_t>(__popc(same));
    }
    __syncthreads();
    // exclusive prefix sum over the experts; before[] becomes the first row of this CTA's pairs of each expert
    {
        const bool has = tid < kDispMaxExperts;                    // whole warps
        const int v = has ? total[tid] + before[tid] : 0;
        int inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += u;
        }
        if (has && lane == 31) scan[warp] = inc;
        __syncthreads();
        if (has) {
            int base = inc - v;
            for (int w = 0; w < warp; ++w) base += scan[w];
            if (blockIdx.x == 0 && blockIdx.y == 0) {
                if (tid < p.n) p.seg[tid] = base;
                if (tid == p.n - 1) p.seg[p.n] = base + v;
            }
            before[tid] += base;
        }
    }
    __syncthreads();
    if (tid < own) {
        int row = -1;
        if (mine >= 0) {
            row = before[mine] + rank_in_warp;
            for (int w = 0; w < warp; ++w) row += in_warp[w][mine];
        }
        own_row[tid] = row;
    }
    __syncthreads();
    int sorted = 0;
    if (tid < own) {
        const int i = tid;
        const int t = static_cast<int>(fast_div(static_cast<uint32_t>(i), p.div_topk)), first = t * topk, e = own_e[i];
        int local = 0;                                             // local rows of the token's pairs before this one
        for (int j = first; j < i; ++j) local += own_row[j] >= 0;
        if (own_row[i] >= 0) to_row[first + local] = own_row[i];
        if (i == first + topk - 1) to_rows[t] = local + (own_row[i] >= 0 ? 1 : 0);
        sorted = first;                                            // place in ascending expert order
        for (int j = first; j < first + topk; ++j) sorted += own_e[j] < e || (own_e[j] == e && j < i);
    }
    __syncthreads();
    if (blockIdx.y == 0 && tid < own) {
        p.pos_sorted[own0 + sorted] = own_row[tid];
        p.w_sorted[own0 + sorted] = p.weights_bf16 ? static_cast<const __nv_bfloat16*>(p.weights)[own0 + tid]
                                                   : __float2bfloat16_rn(static_cast<const float*>(p.weights)[own0 + tid]);
    }
    // quantise: a half-warp per 128-value block, kDispUnroll blocks in flight as long as there are that many.  This kernel is bound by
    // instructions: 32 warps go through every place of a round, whether there is a block or not, and went through all of a
    // token's pairs for every block, local or not.  us before / after: 32 of 256 experts of dim 7168, 4 tokens 5.7 / 5.1, 1024 14.6 / 12.6, 4096
    // 42.6 / 36.8; 20 of 160 of dim 5120, 2048 17.7 / 14.5; 128 of 256, 4096 53.5 / 52.6.
    auto quantise = [&](int i0, auto unroll) {
        constexpr int kU = decltype(unroll)::value;
        uint4 v[kU];
        int tl[kU], bl[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int i = i0 + u * kHalfWarps;
            tl[u] = divide ? i / b_n : static_cast<int>(__umulhi(static_cast<uint32_t>(i), by_b_n));
            bl[u] = b_lo + i - tl[u] * b_n;
            if (i >= items) tl[u] = -1;
            v[u] = kU == 1 && one_round ? early : tl[u] >= 0 ? __ldg(p.x + ((t0 + tl[u]) * nb + bl[u]) * 16 + lane16) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            float m = amax8(v[u]);
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 8));
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 4));
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
            const float sc = scale_from_amax(m, p.scale_fmt);
            if (tl[u] < 0) continue;
            const uint2 q = quant8(v[u], rcp_approx(sc));
            const int64_t t = t0 + tl[u];
            p.xq[(t * nb + bl[u]) * 16 + lane16] = q;
            if (lane16 == 0) p.xs[t * nb + bl[u]] = sc;
            const int rows = to_rows[tl[u]];
            for (int j = 0; j < rows; ++j) {
                const int row = to_row[tl[u] * topk + j];
                p.xq_rows[(static_cast<int64_t>(row) * nb + bl[u]) * 16 + lane16] = q;
                if (lane16 == 0) p.xs_rows[static_cast<int64_t>(bl[u]) * p.P + row] = sc;
            }
        }
    };
    for (int i0 = 0; i0 < items;) {                                // uniform
        if (items - i0 > kHalfWarps) {
            quantise(i0 + (tid >> 4), std::integral_constant<int, kDispUnroll>{});
            i0 += kDispUnroll * kHalfWarps;
        } else {
            quantise(i0 + (tid >> 4), std::integral_constant<int, 1>{});
            i0 += kHalfWarps;
        }
    }
}

// Bookkeeping of the expert loop in one launch (one CTA): groups the (token, expert) pairs by local expert and
// orders every token's pairs by expert id.  Replaces `counts = bincount(indices)`, the per-expert
// `where(indices == i)` (model.py:680-686) and the sort / scan / gather chain a framework needs for the same.
//   seg [n + 1]        : seg[e] = first row of expert e in the grouped order, seg[n] = number of local pairs
//   tok [P]            : token of the pair placed at each row (pairs of other ranks' experts follow seg[n])
//   pair_row [P]       : scratch; row given to pair p, or -1 when its expert is not local
//   pos_sorted, w_sorted [T, topk]: per token, rows and routing weights in ascending expert order
// The order of an expert's rows is whatever the atomics give; with whole tiles (dsv3_fp8_gemm_grouped) every row's result
// depends on that row alone, so the outputs do not depend on it.
constexpr int kRouteThreads = 1024;
constexpr int kRouteMaxExperts = 256;

__global__ void __launch_bounds__(kRouteThreads) moe_route_kernel(const int64_t* __restrict__ indices,
                                                                  const float* __restrict__ weights, int64_t T, int topk,
                                                                  int start, int n, int* __restrict__ seg,
                                                                  int* __restrict__ tok, int* __restrict__ pair_row,
                                                                  int* __restrict__ pos_sorted,
                                                                  __nv_bfloat16* __restrict__ w_sorted) {
    __shared__ int cnt[kRouteMaxExperts + 1];
    __shared__ int cursor[kRouteMaxExperts + 1];
    const int64_t P = T * topk;
    for (int i = threadIdx.x; i <= n; i += kRouteThreads) cnt[i] = 0;
    __syncthreads();
    for (int64_t pr = threadIdx.x; pr < P; pr += kRouteThreads) {
        const int64_t e = indices[pr] - start;
        atomicAdd(&cnt[(e >= 0 && e < n) ? static_cast<int>(e) : n], 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int i = 0; i <= n; ++i) {
            cursor[i] = run;
            if (i <= n) seg[i] = run;
            run += cnt[i];
        }
    }
    __syncthreads();
    for (int64_t pr = threadIdx.x; pr < P; pr += kRouteThreads) {
        const int64_t e = indices[pr] - start;
        const bool local = (e >= 0 && e < n);
        const int row = atomicAdd(&cursor[local ? static_cast<int>(e) : n], 1);
        tok[row] = static_cast<int>(pr / topk);
        pair_row[pr] = local ? row : -1;
    }
    __syncthreads();   // pair_row is read below by other threads of this CTA
    for (int64_t t = threadIdx.x; t < T; t += kRouteThreads) {
        int64_t e[kMaxTopk];
        int order[kMaxTopk];
        for (int j = 0; j < topk; ++j) {          // insertion sort of the token's experts, ascending
            const int64_t ej = indices[t * topk + j];
            int k = j;
            while (k > 0 && e[k - 1] > ej) {
                e[k] = e[k - 1];
                order[k] = order[k - 1];
                --k;
            }
            e[k] = ej;
            order[k] = j;
        }
        for (int j = 0; j < topk; ++j) {
            pos_sorted[t * topk + j] = pair_row[t * topk + order[j]];
            w_sorted[t * topk + j] = __float2bfloat16_rn(weights[t * topk + order[j]]);
        }
    }
}

int check_groups(int n, const void* a, int64_t K) {
    if (n < 1 || n > kMaxGroupsOfTable || K < 16 || K % 16 != 0 || reinterpret_cast<uintptr_t>(a) % 16 != 0) {
        set_last_error("grouped fp8_gemm: needs K %% 16 == 0, a 16-byte aligned a, and 1..%d groups", kMaxGroupsOfTable);
        return DSV3_ERR_UNSUPPORTED;
    }
    return DSV3_OK;
}

StreamSide side_of(const void* a, const float* a_s, bool transposed, int64_t rows, int64_t N, int64_t K) {
    StreamSide d = {};
    d.a = a;
    d.a_s = a_s;
    d.as_row = transposed ? 1 : (K + 127) / 128;
    d.as_chunk = transposed ? rows : 1;
    d.rows = rows;
    d.N = N;
    d.K = K;
    return d;
}

// Tokens per tile for w1 and w3 of an ordinary MLP with SwiGLU and quantisation in one launch, or 0 where no width does: with enough
// weight to keep half of the SMs on whole tiles the launch is a stream of weights up to 128 tokens; beyond, the pair tiles of the
// GEMMs multiply better.  With less it is set-up, epilogue and the chunks of a tile, whole (base + chunk * K chunks) or cut over K as
// the kernel's own plan decides (cut + unit * units), until whole tiles of 128 no longer fit one round.
int swiglu_linear_tile(int64_t M, int64_t N, int64_t K) {
    const int64_t blocks = N / 128, kc = (K + 127) / 128, sms = num_sms();
    if (2 * blocks >= sms) return M <= 16 ? 16 : (M <= 64 ? 64 : (M <= 128 ? 128 : 0));
    struct Cost { int tile; double base, chunk, cut, unit; };
    constexpr Cost kCosts[] = {{16, 4.6, 0.33, 8.9, 0.0030}, {32, 5.8, 0.36, 11.3, 0.0036}, {64, 7.2, 0.46, 17.0, 0.0036}, {128, 7.5, 0.42, 0.0, 0.0}};
    int best = 0;
    double least = 1e30;
    for (const Cost& c : kCosts) {
        const int64_t tiles = blocks * ((M + c.tile - 1) / c.tile);
        if (tiles > sms || tiles * kc >= (1ll << 27)) continue;
        const int units = static_cast<int>(tiles * kc);
        const bool is_cut = cut_ranges(c.tile, static_cast<int>(tiles), units, units, static_cast<int>(kc), units < sms ? units : static_cast<int>(sms)) > 0;
        const double t = is_cut ? c.cut + c.unit * static_cast<double>(tiles * kc) : c.base + c.chunk * static_cast<double>(kc);
        if (t < least) {
            least = t;
            best = c.tile;
        }
    }
    return best;
}

// Whether that is faster on the device than two GEMMs and swiglu_quant.  It is not where its tiles are cut and the GEMMs are at their
// best: up to 8 rows on weights that the decode kernel takes (with few K chunks nothing is cut), and up to 16, 32 and 64 rows on few, or
// on long, rows of weights, which the GEMMs cut inside clusters.  B200, us per MLP in a graph of as many as displace the L2, five
// launches / three: 2048 -> 1408 at 1, 8, 16, 48, 256, 1024 rows 12.0 / 15.0, 13.1 / 15.0, 16.3 / 16.5, 19.3 / 17.3, 22.5 / 19.7, 32.1 /
// 25.6; 1408 -> 2048 at 1, 9, 17 11.8 / 14.6, 16.9 / 16.4, 17.4 / 14.5; 1024 -> 1024 at 1, 8 11.4 / 10.9, 12.6 / 11.0; 4096 -> 1408 at 8,
// 16, 33 16.4 / 18.7, 19.1 / 20.1, 21.6 / 20.1; 7168 -> 1024 at 16, 24, 33 19.4 / 22.6, 20.3 / 20.6, 23.2 / 22.0; 7168 -> 1536 at 1, 8, 33
// 22.1 / 21.1, 21.0 / 21.6, 25.3 / 23.0; 7168 -> 2304 at 1, 16, 24, 48, 256 24.3 / 21.9, 24.3 / 23.0, 25.1 / 26.1, 30.2 / 27.8, 42.0 / 38.1;
// 7168 -> 4608 at 16, 17, 48 32.9 / 31.2, 33.4 / 34.6, 39.7 / 38.3; 7168 -> 512 at 16, 64, 80 17.3 / 19.8, 20.0 / 20.3, 22.2 / 19.0; 5120 ->
// 12288 at 1, 128 44.6 / 41.2, 62.3 / 51.6; 7168 -> 18432 at 1, 16, 128 73.9 / 69.9, 77.9 / 71.7, 102.3 / 90.3.
bool swiglu_linear_faster(int64_t M, int64_t N, int64_t K) {
    const int64_t blocks = N / 128, kc = (K + 127) / 128;
    if (2 * blocks >= num_sms()) return true;
    if (M <= 8 && decode_kernel_pays(M, N, K)) return kc <= 8;
    if (M <= 2) return true;                       // (larger weights at one or two rows: the fused Linear)
    if (M <= 16) return kc <= 24 || blocks >= 16;
    if (M <= 32) return kc <= 40;
    return M > 64 || kc <= 40 || blocks > 6;
}

// The ordinary weight of dsv3_swiglu_gemm_rows / dsv3_fp8_gemm_rows.
int add_ordinary(StreamGemm& q, const dsv3_side_gemm_t* s) {
    if (!s || s->rows == 0 || s->N == 0) return DSV3_OK;
    if (s->rows < 0 || s->N < 0 || s->K < 16 || s->K % 16 != 0 || s->rows >= (1ll << 31) || !s->a || !s->a_s || !s->w || !s->w_s || !s->out ||
        (q.swiglu && (!s->w3 || !s->w3_s || !s->out_s_t || s->N % 128 != 0))) {
        set_last_error("side gemm: null pointer, or sizes outside K %% 16 == 0 (and N %% 128 == 0 with SwiGLU)");
        return DSV3_ERR_INVALID_ARGUMENT;
    }
    if (reinterpret_cast<uintptr_t>(s->a) % 16 || reinterpret_cast<uintptr_t>(s->w) % 16 || reinterpret_cast<uintptr_t>(s->w3) % 16 ||
        reinterpret_cast<uintptr_t>(s->out) % 16) {
        set_last_error("side gemm: a, w, w3 and out must be 16-byte aligned");
        return DSV3_ERR_UNSUPPORTED;
    }
    q.ordinary = side_of(s->a, s->a_s, s->a_s_transposed != 0, s->rows, s->N, s->K);
    q.w0 = s->w;
    q.w0_s = s->w_s;
    q.w1 = s->w3;
    q.w1_s = s->w3_s;
    if (q.swiglu) {
        q.ordinary.hq = s->out;
        q.ordinary.hs = s->out_s_t;
        q.ordinary.hs_row = 1;
        q.ordinary.hs_blk = s->rows;
    } else {
        q.ordinary.c = s->out;
    }
    return DSV3_OK;
}

int grouped_plain(StreamGemm& q, const void* table, int n, const void* a, const float* a_s, bool transposed, const int32_t* seg, int64_t rows_total,
                  int64_t rows_hint, int64_t N, int64_t K, void* c, const dsv3_side_gemm_t* side, void* workspace, size_t workspace_bytes) {
    const int rc = check_groups(n, a, K);
    if (rc != DSV3_OK) return rc;
    q.groups = side_of(a, a_s, transposed, rows_total, N, K);
    q.groups.c = c;
    q.rows_expected = rows_hint > 0 && rows_hint < rows_total ? rows_hint : rows_total;
    q.n_groups = n;
    q.table0 = table;
    q.seg = seg;
    q.workspace = workspace;
    q.workspace_bytes = workspace_bytes;
    return add_ordinary(q, side);
}

}  // namespace

}  // namespace dsv3

using namespace dsv3;

extern "C" {

size_t dsv3_group_table_bytes(int n_groups) { return n_groups > 0 ? group_table_bytes(n_groups) : 0; }

int dsv3_group_table_build(void* table, const void* const* weights, const float* const* scales, int n_groups,
                           int64_t N, int64_t K, dsv3_stream_t stream) {
    if (!table || !weights || !scales || N <= 0 || K <= 0) {
        set_last_error("group_table_build: null pointer or non-positive size");
        return DSV3_ERR_INVALID_ARGUMENT;
    }
    return build_group_table(table, weights, scales, n_groups, N, K, static_cast<cudaStream_t>(stream));
}

int dsv3_fp8_gemm_grouped(const void* table, int n_groups, const void* a, const float* a_s, const int32_t* seg,
                          int64_t rows_total, int64_t rows_hint, int64_t N, int64_t K, void* c, dsv3_stream_t stream) {
    if (rows_total < 0 || rows_hint < 0 || N < 0 || K <= 0) {
        set_last_error("fp8_gemm_grouped: negative size");
        return DSV3_ERR_INVALID_ARGUMENT;
    }
    if (rows_total == 0 || N == 0) return DSV3_OK;
    if (!table || !a || !a_s || !seg || !c) {
        set_last_error("fp8_gemm_grouped: null pointer");
        return DSV3_ERR_INVALID_ARGUMENT;
    }
    StreamGemm q = {};
    const int rc = grouped_plain(q, table, n_groups, a, a_s, false, seg, rows_total, rows_hint, N, K, c, nullptr, nullptr, 0);
    return rc != DSV3_OK ? rc : launch_fp8_stream(q, static_cast<cudaStream_t>(stream));
}

// The arguments of dsv3_fp8_gemm_rows and dsv3_swiglu_gemm_rows as a launch; any: whether there is one.
static int gemm_rows(StreamGemm& q, bool& any, const void* table, int n_groups, const void* a, const float* a_s_t, const int32_t* seg, int64_t rows_total,
                     int64_t rows_hint, int64_t N, int64_t K, void* c, const dsv3_side_gemm_t* side, void* workspace, size_t workspace_bytes) {
    any = false;
    if (rows_total < 0 || rows_hint < 0 || N < 0 || K <= 0) {
        set_last_error("fp8_gemm_rows: negative size");
        return DSV3_ERR_INVALID_ARGUMENT;
    }
    if (rows_total == 0 || N == 0) return DSV3_OK;
    if (!table || !a || !a_s_t || !seg || !c) {
        set_last_error("fp8_gemm_rows: null pointer");
        return DSV3_ERR_INVALID_ARGUMENT;
    }
    any = true;
    return grouped_plain(q, table, n_groups, a, a_s_t, true, seg, rows_total, rows_hint, N, K, c, side, workspace, workspace_bytes);
}

int dsv3_fp8_gemm_rows(const void* table, int n_groups, const void* a, const float* a_s_t, const int32_t* seg, int64_t rows_total,
                       int64_t rows_hint, int64_t N, int64_t K, void* c, const dsv3_side_gemm_t* side, void* workspace,
                       size_t workspace_bytes, dsv3_stream_t stream) {
    StreamGemm q = {};
    bool any = false;
    const int rc = gemm_rows(q, any, table, n_groups, a, a_s_t, seg, rows_total, rows_hint, N, K, c, side, workspace, workspace_bytes);
    return rc != DSV3_OK || !any ? rc : launch_fp8_stream(q, static_cast<cudaStream_t>(stream));
}

static int swiglu_rows(StreamGemm& q, bool& any, const void* table1, const void* table3, int n_groups, const void* a, const float* a_s_t, const int32_t* seg,
                       int64_t rows_total, int64_t rows_hint, int64_t N, int64_t K, int scale_fmt, void* hq, float* hs_t, const dsv3_side_gemm_t* side,
                       void* workspace, size_t workspace_bytes) {
    any = false;
    if (rows_total < 0 || rows_hint < 0 || N < 0 || K <= 0) {
        set_last_error("swiglu_gemm_rows: negative size");
        return DSV3_ERR_INVALID_ARGUMENT;
    }
    if (scale_fmt != DSV3_SCALE_FMT_FP32 && scale_fmt != DSV3_SCALE_FMT_UE8M0) {
        set_last_error("swiglu_gemm_rows: unknown scale_fmt %d", scale_fmt);
        return DSV3_ERR_INVALID_ARGUMENT;
    }
    if (rows_total == 0 || N == 0) return DSV3_OK;
    if (!table1 || !table3 || !a || !a_s_t || !seg || !hq || !hs_t) {
        set_last_error("swiglu_gemm_rows: null pointer");
        return DSV3_ERR_INVALID_ARGUMENT;
    }
    if (N % 128 != 0) {
        set_last_error("swiglu_gemm_rows: N = %lld is not divisible by 128", static_cast<long long>(N));
        return DSV3_ERR_UNSUPPORTED;
    }
    const int rc = check_groups(n_groups, a, K);
    if (rc != DSV3_OK) return rc;
    any = true;
    q.groups = side_of(a, a_s_t, true, rows_total, N, K);
    q.groups.hq = hq;
    q.groups.hs = hs_t;
    q.groups.hs_row = 1;
    q.groups.hs_blk = rows_total;
    q.rows_expected = rows_hint > 0 && rows_hint < rows_total ? rows_hint : rows_total;
    q.n_groups = n_groups;
    q.table0 = table1;
    q.table1 = table3;
    q.seg = seg;
    q.swiglu = true;
    q.scale_fmt = scale_fmt;
    q.workspace = workspace;
    q.workspace_bytes = workspace_bytes;
    return add_ordinary(q, side);
}

int dsv3_swiglu_gemm_rows(const void* table1, const void* table3, int n_groups, const void* a, const float* a_s_t, const int32_t* seg,
                          int64_t rows_total, int64_t rows_hint, int64_t N, int64_t K, int scale_fmt, void* hq, float* hs_t,
                          const dsv3_side_gemm_t* side, void* workspace, size_t workspace_bytes, dsv3_stream_t stream) {
    StreamGemm q = {};
    bool any = false;
    const int rc = swiglu_rows(q, any, table1, table3, n_groups, a, a_s_t, seg, rows_total, rows_hint, N, K, scale_fmt, hq, hs_t, side, workspace, workspace_bytes);
    return rc != DSV3_OK || !any ? rc : launch_fp8_stream(q, static_cast<cudaStream_t>(stream));
}

// The second launch begins to read its weights while the CTAs of the first leave (StreamGemm::early).
int dsv3_expert_gemms(const void* table1, const void* table3, const void* table2, int n_groups, const void* a, const float* a_s_t, const int32_t* seg,
                      int64_t rows_total, int64_t rows_hint, int64_t inter, int64_t dim, int scale_fmt, void* hq, float* hs_t, void* o,
                      const dsv3_side_gemm_t* up, const dsv3_side_gemm_t* down, void* workspace, size_t workspace_bytes, dsv3_stream_t stream) {
    StreamGemm first = {}, second = {};
    bool any_first = false, any_second = false;
    int rc = swiglu_rows(first, any_first, table1, table3, n_groups, a, a_s_t, seg, rows_total, rows_hint, inter, dim, scale_fmt, hq, hs_t, up, workspace,
                         workspace_bytes);
    if (rc == DSV3_OK) rc = gemm_rows(second, any_second, table2, n_groups, hq, hs_t, seg, rows_total, rows_hint, dim, inter, o, down, workspace, workspace_bytes);
    if (rc != DSV3_OK || !any_first || !any_second) return rc;      // (both or neither: rows and sizes are the same)
    first.leads = second.early = true;
    return launch_fp8_streams(first, second, static_cast<cudaStream_t>(stream));
}

// (a kernel or split that the host pinned is one of fp8_gemm's: the separate launches honour or refuse it)
static bool swiglu_linear_serves(int64_t M, int64_t N, int64_t K) {
    return M > 0 && N > 0 && N % 128 == 0 && K >= 128 && K % 128 == 0 && M < (1ll << 31) && gemm_policy_kernel() == 0 && gemm_policy_split() == 0 &&
           swiglu_linear_tile(M, N, K) > 0;
}

int dsv3_swiglu_linear_pays(int64_t M, int64_t N, int64_t K) { return swiglu_linear_serves(M, N, K) && swiglu_linear_faster(M, N, K); }

// Launching three kernels instead of five saves a host 4 to 10 us, of 23 to 30 that it needs for an MLP; up to 24 MB of weights the
// device needs no more than that.  us from Python, five launches / three: 2048 -> 1408 at 1 row 23.5 / 19.6, at 16 30.3 / 20.0; 7168 -> 2304 at
// 24 30.3 / 27.1, 7168 -> 3072 at 17 31.1 / 29.9; but 7168 -> 4608 34.7 / 35.5.
int dsv3_swiglu_linear_saves_launches(int64_t M, int64_t N, int64_t K) { return swiglu_linear_serves(M, N, K) && N * K <= (24ll << 20); }

size_t dsv3_swiglu_linear_workspace_bytes(int64_t M, int64_t N, int64_t K) {
    const int tile = M > 0 && N > 0 && K > 0 ? swiglu_linear_tile(M, N, K) : 0;
    return tile ? stream_tile_workspace_bytes(tile) : 0;
}

int dsv3_swiglu_linear(const void* a, const float* a_s, const void* w1, const float* w1_s, const void* w3, const float* w3_s, int64_t M, int64_t N,
                       int64_t K, int scale_fmt, void* h, float* h_s, void* workspace, size_t workspace_bytes, dsv3_stream_t stream) {
    if (M < 0 || N < 0 || K <= 0) {
        set_last_error("swiglu_linear: negative size");
        return DSV3_ERR_INVALID_ARGUMENT;
    }
    if (scale_fmt != DSV3_SCALE_FMT_FP32 && scale_fmt != DSV3_SCALE_FMT_UE8M0) {
        set_last_error("swiglu_linear: unknown scale_fmt %d", scale_fmt);
        return DSV3_ERR_INVALID_ARGUMENT;
    }
    if (M == 0 || N == 0) return DSV3_OK;
    const dsv3_side_gemm_t side = {a, a_s, 0, M, N, K, w1, w1_s, w3, w3_s, h, h_s};
    StreamGemm q = {};
    q.swiglu = true;
    const int rc = add_ordinary(q, &side);
    if (rc != DSV3_OK) return rc;
    q.ordinary.hs_row = N / 128;                     // as swiglu_quant writes them
    q.ordinary.hs_blk = 1;
    q.scale_fmt = scale_fmt;
    q.tile = swiglu_linear_tile(M, N, K);
    if (q.tile == 0) q.tile = 128;
    q.workspace = workspace;
    q.workspace_bytes = workspace_bytes;
    return launch_fp8_stream(q, static_cast<cudaStream_t>(stream));
}

size_t dsv3_gemm_rows_workspace_bytes(int n_groups, int64_t rows_total, int64_t rows_hint) {
    if (n_groups <= 0 || rows_total <= 0) return 0;
    const int64_t rows = rows_hint > 0 && rows_hint < rows_total ? rows_hint : rows_total;
    return stream_workspace_bytes((rows + n_groups - 1) / n_groups);
}

int dsv3_moe_dispatch(const void* x, int64_t T, int64_t dim, const int64_t* indices, const void* weights, int weights_bf16, int topk,
                      int start, int n_local, int scale_fmt, int32_t* seg, int32_t* pos_sorted, void* w_sorted, void* xq, float* xs,
                      void* xq_rows, float* xs_rows_t, dsv3_stream_t stream) {
    if (T < 0 || topk < 0 || n_local < 0 || dim < 0) {
        set_last_error("moe_dispatch: negative size");
        return DSV3_ERR_INVALID_ARGUMENT;
    }
    if (scale_fmt != DSV3_SCALE_FMT_FP32 && scale_fmt != DSV3_SCALE_FMT_UE8M0) {
        set_last_error("moe_dispatch: unknown scale_fmt %d", scale_fmt);
        return DSV3_ERR_INVALID_ARGUMENT;
    }
    if (T == 0 || topk == 0 || dim == 0) return DSV3_OK;
    if (!x || !indices || !weights || !seg || !pos_sorted || !w_sorted || !xq || !xs || !xq_rows || !xs_rows_t) {
        set_last_error("moe_dispatch: null pointer");
        return DSV3_ERR_INVALID_ARGUMENT;
    }
    if (n_local < 1 || n_local > kDispMaxExperts || topk > kMaxTopk || T * topk >= (1ll << 31) || dim % 128 != 0 || dim > (1 << 24)) {
        set_last_error("moe_dispatch: 1..%d local experts, at most top-%d and 2^31 pairs, dim divisible by 128", kDispMaxExperts, kMaxTopk);
        return DSV3_ERR_UNSUPPORTED;
    }
    if (reinterpret_cast<uintptr_t>(x) % 16 != 0 || reinterpret_cast<uintptr_t>(xq) % 8 != 0 || reinterpret_cast<uintptr_t>(xq_rows) % 8 != 0) {
        set_last_error("moe_dispatch: x must be 16-byte, xq and xq_rows 8-byte aligned");
        return DSV3_ERR_UNSUPPORTED;
    }
    DispatchParams p;
    p.x = static_cast<const uint4*>(x);
    p.indices = indices;
    p.weights = weights;
    p.weights_bf16 = weights_bf16;
    p.T = T;
    p.P = T * topk;
    p.topk = topk;
    p.dim = static_cast<int>(dim);
    p.start = start;
    p.n = n_local;
    p.scale_fmt = scale_fmt;
    p.seg = seg;
    p.pos_sorted = pos_sorted;
    p.w_sorted = static_cast<__nv_bfloat16*>(w_sorted);
    p.xq = static_cast<uint2*>(xq);
    p.xs = xs;
    p.xq_rows = static_cast<uint2*>(xq_rows);
    p.xs_rows = xs_rows_t;
    // one CTA per SM (every CTA counts all pairs), at most kDispPairs own pairs each
    const int64_t wave = num_sms();
    int64_t tpc = (T + wave - 1) / wave;
    if (tpc > kDispPairs / topk) tpc = kDispPairs / topk;
    p.tpc = static_cast<int>(tpc);
    const int64_t gx = (T + tpc - 1) / tpc;
    int gy = 1;                                                    // few tokens: share each token's blocks among CTAs
    while (gy < 8 && gx * gy * 2 <= wave && gy * 2 * 32 <= dim / 128) gy *= 2;
    const int nb = static_cast<int>(dim / 128);
    p.per_y = (nb + gy - 1) / gy;
    const int last = nb - (nb - 1) / p.per_y * p.per_y;
    p.div_topk = make_fast_div(static_cast<uint32_t>(topk));
    p.by_b[0] = 0xFFFFFFFFu / static_cast<uint32_t>(p.per_y) + 1u;
    p.by_b[1] = 0xFFFFFFFFu / static_cast<uint32_t>(last) + 1u;
    DSV3_CUDA_TRY(launch_dependent(moe_dispatch_kernel, dim3(static_cast<unsigned>(gx), static_cast<unsigned>(gy)), dim3(kDispThreads), 0,
                                   static_cast<cudaStream_t>(stream), p));
    return DSV3_OK;
}

int dsv3_moe_route(const int64_t* indices, const float* weights, int64_t T, int topk, int start, int n_local,
                   int32_t* seg, int32_t* tok, int32_t* pair_row, int32_t* pos_sorted, void* w_sorted,
                   dsv3_stream_t stream) {
    if (T < 0 || topk < 0 || n_local < 0) {
        set_last_error("moe_route: negative size");
        return DSV3_ERR_INVALID_ARGUMENT;
    }
    if (n_local > kRouteMaxExperts || topk > kMaxTopk || T * topk >= (1ll << 31)) {
        set_last_error("moe_route: at most %d local experts, top-%d and 2^31 pairs", kRouteMaxExperts, kMaxTopk);
        return DSV3_ERR_UNSUPPORTED;
    }
    if (!seg || (T * topk > 0 && (!indices || !weights || !tok || !pair_row || !pos_sorted || !w_sorted))) {
        set_last_error("moe_route: null pointer");
        return DSV3_ERR_INVALID_ARGUMENT;
    }
    moe_route_kernel<<<1, kRouteThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        indices, weights, T, topk, start, n_local, seg, tok, pair_row, pos_sorted, static_cast<__nv_bfloat16*>(w_sorted));
    DSV3_CUDA_TRY(cudaGetLastError());
    return DSV3_OK;
}

int dsv3_moe_combine(const void* o, const int32_t* pos, const void* w, int64_t T, int topk, int64_t dim, void* y,
                     dsv3_stream_t stream) {
    return dsv3_moe_combine_add(o, pos, w, nullptr, T, topk, dim, y, stream);
}

int dsv3_moe_combine_add(const void* o, const int32_t* pos, const void* w, const void* z, int64_t T, int topk, int64_t dim, void* y,
                         dsv3_stream_t stream) {
    if (T < 0 || topk < 0 || dim < 0) {
        set_last_error("moe_combine: negative size");
        return DSV3_ERR_INVALID_ARGUMENT;
    }
    if (T == 0 || dim == 0) return DSV3_OK;
    if (!pos || !w || !y || (topk > 0 && !o)) {
        set_last_error("moe_combine: null pointer");
        return DSV3_ERR_INVALID_ARGUMENT;
    }
    const bool many = T >= kCombineManyTokens && dim > kCombineManyDim;
    const int64_t cols = dim / 8, pieces = many ? 4 : 1, per_row = (cols + pieces * kThreads - 1) / (pieces * kThreads);
    const int threads = static_cast<int>(((cols + pieces * per_row - 1) / (pieces * per_row) + 31) / 32 * 32);
    if (dim % 8 != 0 || reinterpret_cast<uintptr_t>(o) % 16 != 0 || reinterpret_cast<uintptr_t>(y) % 16 != 0 ||
        reinterpret_cast<uintptr_t>(z) % 16 != 0 || T * per_row >= (1ll << 31)) {
        set_last_error("moe_combine: dim must be a multiple of 8 and o, y (and z) 16-byte aligned");
        return DSV3_ERR_UNSUPPORTED;
    }
    DSV3_CUDA_TRY(launch_dependent(many ? moe_combine_kernel<4, 2> : moe_combine_kernel<1, 6>, dim3(static_cast<unsigned>(T * per_row)), dim3(static_cast<unsigned>(threads)), 0,
                                   static_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16*>(o), pos,
                                   static_cast<const __nv_bfloat16*>(w), static_cast<const __nv_bfloat16*>(z),
                                   static_cast<__nv_bfloat16*>(y), topk, dim, make_fast_div(static_cast<uint32_t>(per_row))));
    return DSV3_OK;
}

}  // extern "C"
