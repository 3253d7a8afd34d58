// Expert layer for a handful of tokens on sm_100a, in two launches: w1 / w3 with SwiGLU, then w2 with the weighted sum.
//
// Replaces MoE.forward's expert loop and shared experts, inference/model.py:683-693 (act_quant, fp8_gemm and SwiGLU per
// expert, :532 / :633), for a decode step of up to eight tokens.
//
// What bounds it: a token's experts are 44 MB each (7168 x 2048), 7 us of HBM; around that, latency.  The four-launch form
// (dispatch, w1 / w3, w2, combine; fp8_stream.cu) cuts the few weight tiles over K to fill the machine, parks the parts in
// global memory and lets the last arrival add them: 12 us a projection for 4.5 and 2.3 us of weights, plus two small
// launches.  Here nothing crosses a CTA:
//   * up: a work item is 16 rows of w1 and the same 16 of w3 over all of K, its eight warps splitting K; one expert of 2048 rows
//     is 128 items, about one per SM, 230 KB each.  A lane's 16-byte loads are the A fragments of mma.sync.m16n8k32 (the K
//     permutation of fp8_linear_small.cu), four chunks of both weights in flight per warp = 128 KB per SM; the next
//     item's loads are issued while the present one is summed up.  Every CTA sorts the (token, expert) pairs and
//     quantises the tokens itself, under its first weight loads.
//   * down: a CTA owns 16 columns of the result and walks over the experts in ascending order, so the weighted bf16 sums
//     of a token (model.py:689) stay in a register; it quantises the rows of h it needs.  dim / 16 CTAs of four warps, four to an SM:
//     resident at once up to 9472 columns and experts 5900 wide, in several rounds beyond.
//   * while `up` sums its last item and `down` is being started HBM would be idle; each CTA asks the L2 for its share of the
//     touched w2 instead.
// B200, one token, one layer of 7168 x 2048 with 32 of 256 experts local, top-8, and an eighth of the shared expert, replayed from
// a graph with cold weights: 30.2 -> 16.1 us (up 11.1 and down 6.3 launched on their own).  The weights go through L1 into
// registers on purpose: past it (L1::no_allocate, cp.async.cg into a ring in shared memory) or with L1 squeezed by more
// shared memory the same layer took 19-22 us.
//
// Arithmetic: per K chunk acc = fma(product * a_s, b_s, acc) (kernel.py:162), warps' sums added in a fixed order; bf16 rounding of
// every GEMM result, of silu, of the product with w3, of the weighted rows and of every partial sum, as the operators round.
#include <cuda.h>

#include "common.cuh"
#include "decode_math.cuh"
#include "gemm_plan.cuh"

namespace dsv3 {

namespace {

constexpr int kMaxTokens = 8;               // the N side of one mma
constexpr int kMaxPairs = 64;
constexpr int kRing = 4;                    // chunks in flight per warp (of each weight)
constexpr int kUpWarps = 8, kUpThreads = kUpWarps * 32;
constexpr int kDownWarps = 4, kDownThreads = kDownWarps * 32;
constexpr int kMaxExperts = kMaxGroupsOfTable;
constexpr int64_t kPrefetchBytes = 48ll << 20;      // of w2, at most (the L2 holds 126 MB)

// The local pairs sorted by (expert, pair); a slot is up to T rows of one expert.
struct Route {
    int n_rows, n_slots;
    int slot_first[kMaxPairs + 1];
    int slot_e[kMaxPairs];
    int row_tok[kMaxPairs];
    float row_w[kMaxPairs];                 // routing weight, rounded to bf16
};

struct UpParams {
    const uint4* x;                         // bf16 [T, dim]
    const int64_t* indices;                 // [T, topk]
    const void* weights;                    // [T, topk], bf16 or fp32
    const uint8_t* const* w1;               // pointers of the n local experts, in device memory
    const uint8_t* const* w3;
    const float* const* s1;
    const float* const* s3;
    const uint8_t* const* w2;
    const uint8_t *sw1, *sw3, *sw2;         // shared experts, or null
    const float *ss1, *ss3;
    __nv_bfloat16* h;                       // [rows of the route][inter]
    __nv_bfloat16* hz;                      // [T][inter_s]
    Route* route;
    int weights_bf16, T, topk, start, n, dim, inter, inter_s, scale_fmt;
};

struct DownParams {
    const Route* route;
    const uint8_t* const* w2;
    const float* const* s2;
    const uint8_t* sw2;                     // shared experts, or null
    const float* ss2;
    const __nv_bfloat16* h;
    const __nv_bfloat16* hz;
    const __nv_bfloat16* z;                 // bf16 [T, dim] to add when there is no sw2, or null
    __nv_bfloat16* y;                       // bf16 [T, dim]
    int T, n, dim, inter, inter_s, scale_fmt;
};

// One chunk of 16 weight rows: rows g and g + 8 of the lane's quad, bytes 16 t .. of both 64-byte halves.
struct Frag {
    uint4 v[4];
    float s;
    // w: the lane's first byte of row g in chunk 0; sc: scale row
    __device__ __forceinline__ void load(const uint8_t* w, int64_t row8, const float* sc, int chunk) {
        const uint8_t* q = w + static_cast<int64_t>(chunk) * kChunkK;
        v[0] = __ldcs(reinterpret_cast<const uint4*>(q));
        v[1] = __ldcs(reinterpret_cast<const uint4*>(q + row8));
        v[2] = __ldcs(reinterpret_cast<const uint4*>(q + 64));
        v[3] = __ldcs(reinterpret_cast<const uint4*>(q + row8 + 64));
        s = __ldg(sc + chunk);
    }
    // acc[0..1]: weight row g, tokens 2t and 2t + 1; acc[2..3]: weight row g + 8
    __device__ __forceinline__ void fold(float (&acc)[4], const uint4& f0, const uint4& f1, float as0, float as1) const {
        float part[4];
        chunk_product(part, v, f0, f1);
        acc[0] = fmaf(part[0] * as0, s, acc[0]);
        acc[1] = fmaf(part[1] * as1, s, acc[1]);
        acc[2] = fmaf(part[2] * as0, s, acc[2]);
        acc[3] = fmaf(part[3] * as1, s, acc[3]);
    }
};

// Tokens of a slot as a lane needs them: row of its B fragment (-1: a column of zeros) and of its two accumulator columns.
struct Cols {
    int b, c0, c1;
    template <typename F>
    __device__ __forceinline__ Cols(int nt, int g, int t, F&& row) {
        b = g < nt ? row(g) : -1;
        c0 = row(min(2 * t, nt - 1));
        c1 = row(min(2 * t + 1, nt - 1));
    }
};

// A half-warp quantises blocks of 128 values: `blocks` of them, from src(block) to (bytes, scale) at dst(block); kUnroll in flight.
template <int kThreads, int kUnroll, typename Src, typename Dst>
__device__ __forceinline__ void quantise_blocks(int blocks, int scale_fmt, Src&& src, Dst&& dst) {
    constexpr int kHalves = kThreads / 16;
    const int l16 = threadIdx.x & 15;
    for (int b0 = (threadIdx.x >> 5) * 2; b0 < blocks; b0 += kUnroll * kHalves) {       // uniform in the warp
        uint4 v[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            const int b = b0 + u * kHalves + ((threadIdx.x >> 4) & 1);
            v[u] = b < blocks ? src(b, l16) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            const int b = b0 + u * kHalves + ((threadIdx.x >> 4) & 1);
            if (b0 + u * kHalves >= blocks) break;                                       // uniform in the warp
            const float sc = half_warp_scale(v[u], scale_fmt);
            if (b < blocks) dst(b, l16, quant8(v[u], rcp_approx(sc)), sc);
        }
    }
}

__global__ void __launch_bounds__(kUpThreads, 1) expert_up_few_kernel(const UpParams p) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ const uint8_t *tw1[kMaxExperts], *tw3[kMaxExperts];
    __shared__ const float *ts1[kMaxExperts], *ts3[kMaxExperts];
    __shared__ Route rt;
    __shared__ __align__(16) int key[kMaxPairs];
    __shared__ int head[kMaxPairs];
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int g = lane >> 2, t = lane & 3;
    const int T = p.T, K = p.dim, kc = K / kChunkK;
    const int row_bytes = K + kRowPad;
    uint8_t* xq = smem;                                                          // [T][row_bytes]
    float* xs = reinterpret_cast<float*>(smem + static_cast<size_t>(T) * row_bytes);   // [T][kc]
    float* red = xs + ((T * kc + 3) & ~3);                                       // [2][kUpWarps][2][T][16]
    const int red_w = 2 * T * 16;

    // the tables were written, and waited for, when they were built
    if (tid < p.n) {
        tw1[tid] = p.w1[tid];
        tw3[tid] = p.w3[tid];
        ts1[tid] = p.s1[tid];
        ts3[tid] = p.s3[tid];
    }
    griddep_wait();
    griddep_launch_dependents();

    // ---- the local pairs in the order (expert, pair)
    const int P = T * p.topk;
    if (tid < kMaxPairs) {
        int k = 0x7fffffff;
        if (tid < P) {
            const int64_t e = __ldg(p.indices + tid) - p.start;
            if (e >= 0 && e < p.n) k = static_cast<int>(e) * kMaxPairs + tid;
        }
        key[tid] = k;
        head[tid] = 0;
    }
    __syncthreads();
    if (tid < kMaxPairs) {
        const int k = key[tid], e = k / kMaxPairs;
        if (k != 0x7fffffff) {
            int rank = 0, within = 0;
            for (int j = 0; j < P; ++j) {
                const int other = key[j];
                rank += other < k;
                within += other < k && other >= e * kMaxPairs;
            }
            rt.row_tok[rank] = tid / p.topk;
            rt.row_w[rank] = p.weights_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(p.weights)[tid])
                                            : __bfloat162float(__float2bfloat16_rn(static_cast<const float*>(p.weights)[tid]));
            head[rank] = within % T == 0 ? e + 1 : 0;
        }
        if (tid == 0) rt.n_rows = 0;
    }
    __syncthreads();
    if (tid < kMaxPairs) {
        // slots begin at the marked rows
        const unsigned m0 = __ballot_sync(0xffffffffu, head[lane] != 0), m1 = __ballot_sync(0xffffffffu, head[32 + lane] != 0);
        if (head[tid] != 0) {
            const unsigned below = (1u << lane) - 1u;
            const int slot = warp == 0 ? __popc(m0 & below) : __popc(m0) + __popc(m1 & below);
            rt.slot_first[slot] = tid;
            rt.slot_e[slot] = head[tid] - 1;
        }
        const unsigned l = __ballot_sync(0xffffffffu, key[tid] != 0x7fffffff);
        if (lane == 0 && l) atomicAdd(&rt.n_rows, __popc(l));
        if (tid == 0) rt.n_slots = __popc(m0) + __popc(m1);
    }
    __syncthreads();
    if (tid == 0) rt.slot_first[rt.n_slots] = rt.n_rows;
    __syncthreads();
    if (blockIdx.x == 0) {                                        // for the next launch
        if (tid < kMaxPairs) {
            p.route->slot_first[tid] = rt.slot_first[tid];
            p.route->slot_e[tid] = rt.slot_e[tid];
            p.route->row_tok[tid] = rt.row_tok[tid];
            p.route->row_w[tid] = rt.row_w[tid];
        }
        if (tid == 0) {
            p.route->slot_first[kMaxPairs] = rt.slot_first[kMaxPairs];
            p.route->n_rows = rt.n_rows;
            p.route->n_slots = rt.n_slots;
        }
    }

    // ---- this CTA's items: 16 rows each, the shared experts' first
    const int n_slots = rt.n_slots, per = p.inter / 16, n_sh = p.sw1 ? p.inter_s / 16 : 0;
    const int n_items = n_sh + n_slots * per;
    const int G = static_cast<int>(gridDim.x), cta = static_cast<int>(blockIdx.x);
    const int lo = static_cast<int>(static_cast<int64_t>(cta) * n_items / G), hi = static_cast<int>(static_cast<int64_t>(cta + 1) * n_items / G);
    // this warp's chunks: n_w of them from c_lo; ring position = chunk number modulo kRing within every item
    const int seg = (kc + kUpWarps - 1) / kUpWarps;
    const int c_lo = warp * seg, n_w = max(0, min(kc - c_lo, seg)), n_pad = (seg + kRing - 1) / kRing * kRing;
    const int64_t row8 = 8 * static_cast<int64_t>(K);
    const uint8_t *a1 = nullptr, *a3 = nullptr;                   // where the next loads come from
    const float *b1 = nullptr, *b3 = nullptr;
    auto source = [&](int item) {
        const uint8_t *w1, *w3;
        int r0;
        if (item < n_sh) {
            r0 = item * 16;
            w1 = p.sw1; w3 = p.sw3; b1 = p.ss1; b3 = p.ss3;
        } else {
            const int k = item - n_sh, slot = k / per, e = rt.slot_e[slot];
            r0 = (k - slot * per) * 16;
            w1 = tw1[e]; w3 = tw3[e]; b1 = ts1[e]; b3 = ts3[e];
        }
        const int64_t off = static_cast<int64_t>(r0 + g) * K + static_cast<int64_t>(c_lo) * kChunkK + 16 * t;
        a1 = w1 + off;
        a3 = w3 + off;
        const int so = (r0 / 128) * kc + c_lo;
        b1 += so;
        b3 += so;
    };
    Frag f1[kRing], f3[kRing];
    if (lo < hi) {
        source(lo);
#pragma unroll
        for (int s = 0; s < kRing; ++s)
            if (s < n_w) {
                f1[s].load(a1, row8, b1, s);
                f3[s].load(a3, row8, b3, s);
            }
        quantise_blocks<kUpThreads, 4>(T * kc, p.scale_fmt, [&](int b, int l) { return __ldg(p.x + static_cast<int64_t>(b) * 16 + l); },
                                       [&](int b, int l, uint2 q, float sc) {
                                           const int tok = b / kc, c = b - tok * kc;
                                           *reinterpret_cast<uint2*>(xq + tok * row_bytes + c * kChunkK + l * 8) = q;
                                           if (l == 0) xs[b] = sc;
                                       });
    }
    __syncthreads();

    for (int item = lo; item < hi; ++item) {
        const bool shared = item < n_sh;
        const int slot = shared ? 0 : (item - n_sh) / per;
        const int first = shared ? 0 : rt.slot_first[slot];
        const int nt = shared ? T : rt.slot_first[slot + 1] - first;
        const Cols col(nt, g, t, [&](int i) { return shared ? i : rt.row_tok[first + i]; });
        const uint8_t* xr = xq + max(col.b, 0) * row_bytes + c_lo * kChunkK + 16 * t;
        const float *as0 = xs + col.c0 * kc + c_lo, *as1 = xs + col.c1 * kc + c_lo;
        float acc1[4] = {0.0f, 0.0f, 0.0f, 0.0f}, acc3[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        for (int i0 = 0; i0 < n_pad; i0 += kRing) {
            const bool last = i0 + kRing >= n_pad;
            if (last && item + 1 < hi) source(item + 1);
#pragma unroll
            for (int s = 0; s < kRing; ++s) {
                const int c = i0 + s;
                if (c < n_w) {
                    uint4 x0 = make_uint4(0u, 0u, 0u, 0u), x1 = x0;
                    if (col.b >= 0) {
                        x0 = *reinterpret_cast<const uint4*>(xr + c * kChunkK);
                        x1 = *reinterpret_cast<const uint4*>(xr + c * kChunkK + 64);
                    }
                    f1[s].fold(acc1, x0, x1, as0[c], as1[c]);
                    f3[s].fold(acc3, x0, x1, as0[c], as1[c]);
                }
                const int nc = last ? s : c + kRing;
                if (nc < n_w && !(last && item + 1 >= hi)) {
                    f1[s].load(a1, row8, b1, nc);
                    f3[s].load(a3, row8, b3, nc);
                }
            }
        }
        // the warps' sums; the buffer alternates, so one barrier per item is enough
        float* buf = red + ((item - lo) & 1) * (kUpWarps * red_w);
        float* mine = buf + warp * red_w + 2 * t * 16 + g;
        if (2 * t < nt) {
            mine[0] = acc1[0]; mine[8] = acc1[2];
            mine[T * 16] = acc3[0]; mine[T * 16 + 8] = acc3[2];
        }
        if (2 * t + 1 < nt) {
            mine[16] = acc1[1]; mine[24] = acc1[3];
            mine[T * 16 + 16] = acc3[1]; mine[T * 16 + 24] = acc3[3];
        }
        __syncthreads();
        const int tok = tid >> 4, r = tid & 15;
        if (tok < nt) {
            float h1 = 0.0f, h3 = 0.0f;
#pragma unroll
            for (int w = 0; w < kUpWarps; ++w) {
                h1 += buf[w * red_w + tid];
                h3 += buf[w * red_w + T * 16 + tid];
            }
            const float a = __bfloat162float(__float2bfloat16_rn(h1)), b = __bfloat162float(__float2bfloat16_rn(h3));
            const __nv_bfloat16 h = __float2bfloat16_rn(silu_exact(a) * b);
            if (shared) p.hz[static_cast<int64_t>(tok) * p.inter_s + item * 16 + r] = h;
            else p.h[static_cast<int64_t>(first + tok) * p.inter + (item - n_sh - slot * per) * 16 + r] = h;
        }
    }

    // ---- w2 of the touched experts (and the shared ones') on its way into the L2
    {
        const int64_t bytes = static_cast<int64_t>(K) * p.inter, bytes_s = p.sw1 ? static_cast<int64_t>(K) * p.inter_s : 0;
        const int n_pre = static_cast<int>(min(static_cast<int64_t>(n_slots), kPrefetchBytes / bytes));
        const int s = tid - (bytes_s > 0 ? 1 : 0);
        if (s < n_pre && (s < 0 || s == 0 || rt.slot_e[s] != rt.slot_e[s - 1])) {
            const uint8_t* w = s < 0 ? p.sw2 : p.w2[rt.slot_e[s]];
            const int64_t n16 = (s < 0 ? bytes_s : bytes) / 16;
            int64_t at = n16 * cta / G * 16;
            const int64_t end = n16 * (cta + 1) / G * 16;
            while (at < end) {
                const uint32_t piece = static_cast<uint32_t>(min(end - at, static_cast<int64_t>(16384)));
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(w + at), "r"(piece) : "memory");
                at += piece;
            }
        }
    }
}

__global__ void __launch_bounds__(kDownThreads, 4) expert_down_few_kernel(const DownParams p) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ const uint8_t* tw2[kMaxExperts];
    __shared__ const float* ts2[kMaxExperts];
    __shared__ Route rt;
    __shared__ float red[kDownWarps][kMaxTokens][16];
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int g = lane >> 2, t = lane & 3;
    const int T = p.T;
    const int r0 = static_cast<int>(blockIdx.x) * 16;             // columns of the result = rows of w2
    const int widest = max(p.inter, p.sw2 ? p.inter_s : 0);
    const int row_bytes = widest + kRowPad;
    uint8_t* hq = smem;                                           // [kMaxTokens][row_bytes]
    float* hs = reinterpret_cast<float*>(smem + kMaxTokens * row_bytes);      // [kMaxTokens][widest / 128]
    const int hs_row = widest / kChunkK;

    for (int i = tid; i < p.n; i += kDownThreads) {
        tw2[i] = p.w2[i];
        ts2[i] = p.s2[i];
    }
    griddep_launch_dependents();
    griddep_wait();
    if (tid < kMaxPairs) {
        rt.slot_first[tid] = p.route->slot_first[tid];
        rt.slot_e[tid] = p.route->slot_e[tid];
        rt.row_tok[tid] = p.route->row_tok[tid];
        rt.row_w[tid] = p.route->row_w[tid];
    } else if (tid == kMaxPairs) {
        rt.slot_first[kMaxPairs] = p.route->slot_first[kMaxPairs];
        rt.n_slots = p.route->n_slots;
    }
    __syncthreads();
    const int routed = rt.n_slots, n_slots = routed + (p.sw2 ? 1 : 0);        // the shared experts come last

    auto quantise_rows = [&](const __nv_bfloat16* h, int n, int K) {
        const int kc = K / kChunkK;
        quantise_blocks<kDownThreads, 4>(n * kc, p.scale_fmt,
                                         [&](int blk, int l) { return __ldg(reinterpret_cast<const uint4*>(h) + static_cast<int64_t>(blk) * 16 + l); },
                                         [&](int blk, int l, uint2 q, float sc) {
                                             const int row = blk / kc, c = blk - row * kc;
                                             *reinterpret_cast<uint2*>(hq + row * row_bytes + c * kChunkK + l * 8) = q;
                                             if (l == 0) hs[row * hs_row + c] = sc;
                                         });
    };
    // this warp's chunks of a slot, and where they come from
    int c_lo = 0, n_w = 0, n_pad = 0;
    int64_t row8 = 0;
    const uint8_t* a = nullptr;
    const float* b = nullptr;
    auto source = [&](int slot) {
        const int K = slot < routed ? p.inter : p.inter_s;
        const uint8_t* w = slot < routed ? tw2[rt.slot_e[slot]] : p.sw2;
        const float* s = slot < routed ? ts2[rt.slot_e[slot]] : p.ss2;
        const int kc = K / kChunkK;
        const int seg = (kc + kDownWarps - 1) / kDownWarps;
        c_lo = warp * seg;
        n_w = max(0, min(kc - c_lo, seg));
        n_pad = (seg + kRing - 1) / kRing * kRing;
        row8 = 8 * static_cast<int64_t>(K);
        a = w + static_cast<int64_t>(r0 + g) * K + static_cast<int64_t>(c_lo) * kChunkK + 16 * t;
        b = s + static_cast<int64_t>(r0 / 128) * kc + c_lo;
    };
    Frag f[kRing];
    if (n_slots > 0) {
        source(0);
#pragma unroll
        for (int s = 0; s < kRing; ++s)
            if (s < n_w) f[s].load(a, row8, b, s);
    }
    float y = 0.0f;                                               // token tid / 16, column tid % 16
    const int my_tok = tid >> 4;
    for (int slot = 0; slot < n_slots; ++slot) {
        const bool shared = slot >= routed;
        const int first = shared ? 0 : rt.slot_first[slot];
        const int nt = shared ? T : rt.slot_first[slot + 1] - first;
        const int n_now = n_w, pad_now = n_pad, c_now = c_lo;
        // (the rows before have been read by everyone: the barrier behind the sums)
        quantise_rows(shared ? p.hz : p.h + static_cast<int64_t>(first) * p.inter, nt, shared ? p.inter_s : p.inter);
        __syncthreads();
        const Cols col(nt, g, t, [](int i) { return i; });
        const uint8_t* xr = hq + max(col.b, 0) * row_bytes + c_now * kChunkK + 16 * t;
        const float *as0 = hs + col.c0 * hs_row + c_now, *as1 = hs + col.c1 * hs_row + c_now;
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        for (int i0 = 0; i0 < pad_now; i0 += kRing) {
            const bool last = i0 + kRing >= pad_now;
            if (last && slot + 1 < n_slots) source(slot + 1);     // from here on n_w, a, b are the next slot's
#pragma unroll
            for (int s = 0; s < kRing; ++s) {
                const int c = i0 + s;
                if (c < n_now) {
                    uint4 x0 = make_uint4(0u, 0u, 0u, 0u), x1 = x0;
                    if (col.b >= 0) {
                        x0 = *reinterpret_cast<const uint4*>(xr + c * kChunkK);
                        x1 = *reinterpret_cast<const uint4*>(xr + c * kChunkK + 64);
                    }
                    f[s].fold(acc, x0, x1, as0[c], as1[c]);
                }
                const int nc = last ? s : c + kRing;
                if (nc < n_w && !(last && slot + 1 >= n_slots)) f[s].load(a, row8, b, nc);
            }
        }
        float* mine = &red[warp][0][0] + 2 * t * 16 + g;
        if (2 * t < nt) { mine[0] = acc[0]; mine[8] = acc[2]; }
        if (2 * t + 1 < nt) { mine[16] = acc[1]; mine[24] = acc[3]; }
        __syncthreads();
        // a token's rows of this slot (more than one where an expert is listed twice), in the order of the pairs
        for (int q = 0; q < nt; ++q) {
            if ((shared ? q : rt.row_tok[first + q]) != my_tok) continue;
            float sum = 0.0f;
#pragma unroll
            for (int w = 0; w < kDownWarps; ++w) sum += red[w][q][tid & 15];
            const float o = __bfloat162float(__float2bfloat16_rn(sum));
            if (shared) y += o;
            else y = __bfloat162float(__float2bfloat16_rn(y + __bfloat162float(__float2bfloat16_rn(o * rt.row_w[first + q]))));
        }
    }
    if (my_tok < T) {
        const int64_t at = static_cast<int64_t>(my_tok) * p.dim + r0 + (tid & 15);
        if (p.z) y += __bfloat162float(p.z[at]);
        p.y[at] = __float2bfloat16_rn(y);
    }
}

int up_smem(int64_t T, int64_t dim) {
    return static_cast<int>(T * (dim + kRowPad) + ((T * (dim / kChunkK) + 3) & ~3ll) * 4 + 2 * kUpWarps * 2 * T * 16 * 4);
}
int down_smem(int64_t widest) { return static_cast<int>(kMaxTokens * (widest + kRowPad) + kMaxTokens * (widest / kChunkK) * 4); }

constexpr int kMaxUpSmem = 160 * 1024, kMaxDownSmem = 96 * 1024;

// The kernel is given the largest size there is, whatever this call needs: threads whose first calls differ set the same.
template <typename P>
int launch(void (*kern)(P), int grid, int threads, int smem, int max_smem, const P& prm, cudaStream_t stream, bool (&configured)[64]) {
    int dev = 0;
    DSV3_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) {
        set_last_error("expert layer: device ordinal %d is outside the supported range", dev);
        return DSV3_ERR_UNSUPPORTED;
    }
    if (!configured[dev]) {
        DSV3_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem));
        configured[dev] = true;
    }
    DSV3_CUDA_TRY(launch_dependent(kern, dim3(static_cast<unsigned>(grid)), dim3(threads), static_cast<size_t>(smem), stream, prm));
    return DSV3_OK;
}

// What the two kernels can do; whether they pay is few_experts_pay's business.
bool supported(int64_t T, int topk, int n, int64_t dim, int64_t inter, int64_t inter_s) {
    return T >= 1 && T <= kMaxTokens && topk >= 1 && topk <= kMaxTopk && T * topk <= kMaxPairs && n >= 1 && n <= kMaxExperts &&
           dim >= 128 && dim % 128 == 0 && inter >= 128 && inter % 128 == 0 && inter_s >= 0 && inter_s % 128 == 0 && dim < (1 << 20) && inter < (1 << 20) && inter_s < (1 << 20) &&
           up_smem(T, dim) <= kMaxUpSmem && down_smem(inter > inter_s ? inter : inter_s) <= kMaxDownSmem;
}

bool aligned16(const void* q) { return reinterpret_cast<uintptr_t>(q) % 16 == 0; }

}  // namespace

}  // namespace dsv3

using namespace dsv3;

extern "C" {

int dsv3_few_experts_pay(int64_t T, int topk, int n_local, int64_t n_routed, int64_t dim, int64_t inter, int64_t inter_shared) {
    // Up to two local pairs on average.  Both launches walk over the experts one after the other and lose time at every one of
    // them, and the rows of more tokens take L1 from the weight streams; the tiles of fp8_stream.cu stream many experts at the
    // copy rate but cost 25 us around that.  B200, us, layers with cold weights and unlike routing replayed from a graph (mean), here
    // / in four launches, by expected pairs: 7168 x 2048, 32 of 256 experts: 1 18.5 / 29.6, 2 21.9 / 33.7, 3 26.0 / 37.3, 4 30.6 / 39.3, 6
    // 49.0 / 48.7; all 256: 8 82 / 80.  5120 x 1536, 20 of 160: 0.75 15.0 / 28.3, 1.5 22.2 / 32.1, 3 30.7 / 35.0.  2048 x 1408, 16 of 64:
    // 1.5 15.1 / 28.7, 3 21.6 / 28.5, 6 32.2 / 29.0.  On average the two launches are ahead up to four pairs; a step with more
    // touched experts than that loses, and with two expected such steps are rare.
    // Not under an SM budget: `down` is one small CTA per 16 columns, which spread over all SMs.
    if (!supported(T, topk, n_local, dim, inter, inter_shared) || sm_budget_set()) return 0;
    return T * topk * n_local <= 2 * (n_routed > n_local ? n_routed : n_local);
}

size_t dsv3_few_route_bytes(void) { return sizeof(Route); }

int dsv3_few_up(const void* table1, const void* table3, const void* table2, int n, const void* x, int64_t T, int64_t dim, const int64_t* indices,
                const void* weights, int weights_bf16, int topk, int start, int64_t inter, int scale_fmt, void* route, void* h,
                const dsv3_few_shared_t* shared, dsv3_stream_t stream) {
    const int64_t inter_s = shared ? shared->inter : 0;
    if (!table1 || !table3 || !table2 || !x || !indices || !weights || !route || !h ||
        (shared && (!shared->w1 || !shared->w3 || !shared->w2 || !shared->w1_s || !shared->w3_s || !shared->w2_s || !shared->h || inter_s <= 0))) {
        set_last_error("few_up: null pointer");
        return DSV3_ERR_INVALID_ARGUMENT;
    }
    if (scale_fmt != DSV3_SCALE_FMT_FP32 && scale_fmt != DSV3_SCALE_FMT_UE8M0) {
        set_last_error("few_up: unknown scale_fmt %d", scale_fmt);
        return DSV3_ERR_INVALID_ARGUMENT;
    }
    if (!supported(T, topk, n, dim, inter, inter_s) || !aligned16(x) || !aligned16(h) ||
        (shared && (!aligned16(shared->w1) || !aligned16(shared->w3) || !aligned16(shared->w2) || !aligned16(shared->h)))) {
        set_last_error("few_up: 1..%d tokens, at most top-%d, %d pairs and %d experts, sizes divisible by 128, 16-byte alignment", kMaxTokens, kMaxTopk,
                       kMaxPairs, kMaxExperts);
        return DSV3_ERR_UNSUPPORTED;
    }
    UpParams p = {};
    p.x = static_cast<const uint4*>(x);
    p.indices = indices;
    p.weights = weights;
    p.w1 = table_weights(table1, n);
    p.w3 = table_weights(table3, n);
    p.w2 = table_weights(table2, n);
    p.s1 = table_scales(table1, n);
    p.s3 = table_scales(table3, n);
    if (shared) {
        p.sw1 = static_cast<const uint8_t*>(shared->w1);
        p.sw3 = static_cast<const uint8_t*>(shared->w3);
        p.sw2 = static_cast<const uint8_t*>(shared->w2);
        p.ss1 = shared->w1_s;
        p.ss3 = shared->w3_s;
        p.hz = static_cast<__nv_bfloat16*>(shared->h);
    }
    p.h = static_cast<__nv_bfloat16*>(h);
    p.route = static_cast<Route*>(route);
    p.weights_bf16 = weights_bf16;
    p.T = static_cast<int>(T);
    p.topk = topk;
    p.start = start;
    p.n = n;
    p.dim = static_cast<int>(dim);
    p.inter = static_cast<int>(inter);
    p.inter_s = static_cast<int>(inter_s);
    p.scale_fmt = scale_fmt;
    static bool configured[64] = {};
    // one CTA per SM, and no more than there can be items
    const int64_t most = (inter_s + (T * topk < n ? T * topk : n + topk) * inter) / 16;
    const int grid = static_cast<int>(most < num_sms() ? most : num_sms());
    return launch(expert_up_few_kernel, grid, kUpThreads, up_smem(T, dim), kMaxUpSmem, p, static_cast<cudaStream_t>(stream), configured);
}

int dsv3_few_down(const void* table2, int n, const void* route, const void* h, int64_t T, int topk, int64_t dim, int64_t inter, int scale_fmt,
                  const dsv3_few_shared_t* shared, const void* z, void* y, dsv3_stream_t stream) {
    const int64_t inter_s = shared ? shared->inter : 0;
    if (!table2 || !route || !h || !y || (shared && (!shared->w2 || !shared->w2_s || !shared->h || inter_s <= 0)) || (shared && z)) {
        set_last_error("few_down: null pointer, or both shared experts and z");
        return DSV3_ERR_INVALID_ARGUMENT;
    }
    if (scale_fmt != DSV3_SCALE_FMT_FP32 && scale_fmt != DSV3_SCALE_FMT_UE8M0) {
        set_last_error("few_down: unknown scale_fmt %d", scale_fmt);
        return DSV3_ERR_INVALID_ARGUMENT;
    }
    if (!supported(T, topk, n, dim, inter, inter_s) || !aligned16(h) || !aligned16(z) || (shared && (!aligned16(shared->w2) || !aligned16(shared->h)))) {
        set_last_error("few_down: 1..%d tokens, at most top-%d, %d pairs and %d experts, sizes divisible by 128, 16-byte alignment", kMaxTokens, kMaxTopk,
                       kMaxPairs, kMaxExperts);
        return DSV3_ERR_UNSUPPORTED;
    }
    DownParams p = {};
    p.route = static_cast<const Route*>(route);
    p.w2 = table_weights(table2, n);
    p.s2 = table_scales(table2, n);
    if (shared) {
        p.sw2 = static_cast<const uint8_t*>(shared->w2);
        p.ss2 = shared->w2_s;
        p.hz = static_cast<const __nv_bfloat16*>(shared->h);
    }
    p.h = static_cast<const __nv_bfloat16*>(h);
    p.z = static_cast<const __nv_bfloat16*>(z);
    p.y = static_cast<__nv_bfloat16*>(y);
    p.T = static_cast<int>(T);
    p.n = n;
    p.dim = static_cast<int>(dim);
    p.inter = static_cast<int>(inter);
    p.inter_s = static_cast<int>(inter_s);
    p.scale_fmt = scale_fmt;
    static bool configured[64] = {};
    return launch(expert_down_few_kernel, static_cast<int>(dim / 16), kDownThreads, down_smem(inter > inter_s ? inter : inter_s), kMaxDownSmem, p,
                  static_cast<cudaStream_t>(stream), configured);
}

}  // extern "C"
