// Decode-sized Linear for sm_100a (at most 16 token rows): act_quant folded into the GEMM, one launch.
//
// Replaces the FP8 branch of linear(), inference/model.py:158-160 (act_quant, kernel.py:38-57, followed by
// fp8_gemm, kernel.py:175-196), for the rows of one decode step.  With a handful of tokens the Linear is a stream
// of weight bytes; what it costs beyond that stream is fixed overhead, and the two-launch form pays it twice and
// sends the FP8 activations through HBM in between.  The tcgen05 kernels also carry set-up this regime cannot
// amortise over 2-15 MB of weights (TMEM allocation, tensor maps, mbarrier rings, a split-K workspace with
// tickets).  This kernel has none of it:
//
//   * a warp owns 16 weight rows and a range of 128-wide K chunks; every lane fetches 16 contiguous bytes of a
//     row straight into registers (ld.global, four chunks in flight per warp), which IS the A fragment of
//     mma.sync.m16n8k32 (e4m3 x e4m3 -> fp32) once the K positions inside a 64-byte slab are permuted the same way
//     for both operands (lane t of a quad holds bytes 16t..16t+15: the first mma takes bytes 0-7, the second 8-15);
//   * the token rows (8 or 16, zero-padded) are the N side of the mma.  The CTA quantises its K range of the
//     activations once, bit-identically to act_quant (same arithmetic, quant_math.cuh), into shared memory, or
//     copies already quantised activations there; the fragments are 16-byte shared-memory loads;
//   * every chunk's product is scaled as the reference does, acc = fma(p * a_s, b_s, acc) (kernel.py:162);
//   * K is split over the warps of a CTA and over the CTAs of a cluster (at most 8); partial sums meet in the
//     CTA's shared memory and then in that of the cluster's first CTA (st.shared::cluster), added in a fixed order,
//     so the result is deterministic and no global scratch or atomics are involved.
//
// No wait in this kernel can hang: the only synchronisation is __syncthreads and the cluster barrier, which every
// thread reaches unconditionally.
#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "decode_math.cuh"
#include "gemm_plan.cuh"

namespace dsv3 {

namespace {

constexpr int kRing = 4;        // weight chunks in flight per warp (16 x 16-byte loads per lane)

struct SmallParams {
    const uint4* x;          // bf16 [M, K], 8 values per uint4 (quantised here)       -- or nullptr
    const uint8_t* a;        // e4m3 [M, K], already quantised                         -- used when x is null
    const float* a_s;        // fp32 [M, kc]
    const uint8_t* w;        // e4m3 [N, K]
    const float* w_s;        // fp32 [ceil(N/128), kc]
    __nv_bfloat16* c;        // bf16 [M, N]
    int M, N, K, kc;
    int cpc;                 // K chunks per CTA of a cluster
    int csize;               // CTAs per cluster (K splits across CTAs)
    int scale_fmt;
};

__device__ __forceinline__ void prefetch_l2(const void* ptr) { asm volatile("prefetch.global.L2 [%0];" ::"l"(ptr)); }

__device__ __forceinline__ void st_cluster_f32x4(uint32_t addr_cluster, float4 v) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr_cluster), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

constexpr size_t align16(size_t v) { return (v + 15) & ~static_cast<size_t>(15); }

constexpr size_t kMaxSmem = 200 * 1024;      // of a CTA: the staged activations, scales and partial sums

// WR x WK warps: WR row tiles of 16 weight rows per CTA, WK warps share a row tile and split the CTA's K range.
// MT: token groups of 8 (1 or 2).  kFused: activations arrive as bf16 and are quantised here.
template <int WR, int WK, int MT, bool kFused>
__global__ void __launch_bounds__(WR * WK * 32) fp8_linear_small_kernel(const SmallParams p) {
    constexpr int kThreads = WR * WK * 32;
    constexpr int TOK = 8 * MT;
    extern __shared__ __align__(16) uint8_t smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const uint32_t rank = cluster_ctarank();
    const int rowgroup = static_cast<int>(blockIdx.x) / p.csize;
    const int wr = warp / WK, wk = warp % WK;
    const int r0 = (rowgroup * WR + wr) * 16;
    const int N = p.N, K = p.K, kc = p.kc, cpc = p.cpc;
    const int c0 = static_cast<int>(rank) * cpc;
    const int c1 = min(kc, c0 + cpc);
    const int n_cta = max(c1 - c0, 0);                   // chunks of this CTA
    const int seg = (n_cta + WK - 1) / WK;
    const int w0 = c0 + wk * seg;
    const int n_w = max(min(c1, w0 + seg) - w0, 0);      // chunks of this warp: [w0, w0 + n_w)

    const int row_bytes = cpc * kChunkK + kRowPad;
    uint8_t* xq_s = smem;                                                        // [TOK][row_bytes]
    float* xs_s = reinterpret_cast<float*>(smem + align16(static_cast<size_t>(TOK) * row_bytes));   // [TOK][cpc]
    float* bs_s = xs_s + TOK * cpc;                                              // [WR][cpc]
    float* slots = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bs_s) + align16(static_cast<size_t>(WR) * cpc * 4));
    // partial sums: slots [WK][TOK][ROWS] of this CTA's warps, then [csize][TOK][ROWS] of the CTAs (the cluster's first one)
    constexpr int ROWS = WR * 16;
    float* gathered = slots + WK * TOK * ROWS;

    // rows of this lane (clamped at the edge: the loads stay inside the matrix, the results are masked)
    const uint8_t* wa = p.w + static_cast<int64_t>(min(r0 + g, N - 1)) * K + 16 * t;
    const uint8_t* wb = p.w + static_cast<int64_t>(min(r0 + g + 8, N - 1)) * K + 16 * t;
    // Programmatic dependent launch: the weights are constants of the model, so pulling this warp's first chunks
    // into L2 may overlap the tail of the kernel that produces the activations (L2 is the point of coherence: if
    // that kernel were still writing the weights, the loads after the wait would see its data all the same).
    griddep_launch_dependents();
    if (p.csize > 1) cluster_arrive();        // waited for before the first store into the first CTA's shared memory
    if (t == 0) {
        for (int s = 0; s < kRing && s < n_w; ++s) {
            prefetch_l2(wa + static_cast<int64_t>(w0 + s) * kChunkK);
            prefetch_l2(wb + static_cast<int64_t>(w0 + s) * kChunkK);
        }
    }
    griddep_wait();

    const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);
    auto load_chunk = [&](uint4 (&buf)[4], int c) {
        const int64_t off = static_cast<int64_t>(c) * kChunkK;
        const int k = c * kChunkK + 16 * t;                  // K % 16 == 0: a 16-byte piece is inside or outside
        const bool in0 = k + 16 <= K, in1 = k + 64 + 16 <= K;
        buf[0] = in0 ? __ldcs(reinterpret_cast<const uint4*>(wa + off)) : zero4;
        buf[1] = in0 ? __ldcs(reinterpret_cast<const uint4*>(wb + off)) : zero4;
        buf[2] = in1 ? __ldcs(reinterpret_cast<const uint4*>(wa + off + 64)) : zero4;
        buf[3] = in1 ? __ldcs(reinterpret_cast<const uint4*>(wb + off + 64)) : zero4;
    };
    uint4 ring[kRing][4];
#pragma unroll
    for (int s = 0; s < kRing; ++s)
        if (s < n_w) load_chunk(ring[s], w0 + s);

    // ---- the CTA's K range of the activations: FP8 bytes and scales into shared memory
    if constexpr (kFused) {
        // a half-warp per (token, chunk) block: 16 lanes x 8 bf16, as in the stand-alone act_quant kernel, kBlocks of them
        // requested at once (each round is a trip to L2) and worked on side by side: blocks beyond the last go along as zeros,
        // since a branch between the blocks would put their chains of shuffles one behind the other (7168 -> 1536 at 2 and 4
        // tokens 7.5 / 8.8 us with it, 7.0 / 8.2 without)
        constexpr int kHalves = kThreads / 16;
        const int l16 = threadIdx.x & 15;
        const int nblk = p.M * n_cta;
        auto quantise = [&](auto blocks) {
            constexpr int kBlocks = decltype(blocks)::value;
            for (int b0 = (threadIdx.x >> 5) * 2; b0 < nblk; b0 += kBlocks * kHalves) {     // warp-uniform trip count
                uint4 v[kBlocks];
                int m[kBlocks], cl[kBlocks];
#pragma unroll
                for (int i = 0; i < kBlocks; ++i) {
                    const int b = b0 + i * kHalves + ((threadIdx.x >> 4) & 1);
                    m[i] = b < nblk ? (p.M == 1 ? 0 : b / n_cta) : -1;
                    cl[i] = m[i] >= 0 ? b - m[i] * n_cta : 0;
                    v[i] = m[i] >= 0 ? __ldg(p.x + (static_cast<int64_t>(m[i]) * K + static_cast<int64_t>(c0 + cl[i]) * kChunkK) / 8 + l16) : zero4;
                }
#pragma unroll
                for (int i = 0; i < kBlocks; ++i) {
                    const float sc = half_warp_scale(v[i], p.scale_fmt);
                    if (m[i] >= 0) {
                        *reinterpret_cast<uint2*>(xq_s + m[i] * row_bytes + cl[i] * kChunkK + l16 * 8) = quant8(v[i], rcp_approx(sc));
                        if (l16 == 0) xs_s[m[i] * cpc + cl[i]] = sc;
                    }
                }
            }
        };
        if (nblk <= kHalves) quantise(std::integral_constant<int, 1>{});
        else quantise(std::integral_constant<int, 4>{});
    } else {
        // already quantised activations: asynchronous 16-byte copies, all in flight at once
        const int pieces = n_cta * (kChunkK / 16);               // 16-byte pieces per token row
        const uint32_t xq0 = smem_u32(xq_s);
        for (int idx = threadIdx.x; idx < p.M * pieces; idx += kThreads) {
            const int m = idx / pieces, pc = idx - m * pieces;
            const int k = c0 * kChunkK + pc * 16;
            if (k + 16 <= K) {
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(xq0 + m * row_bytes + pc * 16),
                             "l"(p.a + static_cast<int64_t>(m) * K + k)
                             : "memory");
            } else {
                *reinterpret_cast<uint4*>(xq_s + m * row_bytes + pc * 16) = zero4;
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        for (int idx = threadIdx.x; idx < p.M * n_cta; idx += kThreads) {
            const int m = idx / n_cta, cl = idx - m * n_cta;
            xs_s[m * cpc + cl] = __ldg(p.a_s + static_cast<int64_t>(m) * kc + c0 + cl);
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    // token rows beyond M multiply as zeros
    {
        const int pieces = n_cta * (kChunkK / 16);
        for (int idx = threadIdx.x; idx < (TOK - p.M) * pieces; idx += kThreads) {
            const int m = p.M + idx / pieces, pc = idx % pieces;
            *reinterpret_cast<uint4*>(xq_s + m * row_bytes + pc * 16) = zero4;
        }
        for (int idx = threadIdx.x; idx < (TOK - p.M) * n_cta; idx += kThreads)
            xs_s[(p.M + idx / n_cta) * cpc + idx % n_cta] = 0.0f;
    }
    // weight scales of the CTA's row tiles (a 16-row tile lies inside one 128-row scale block)
    for (int idx = threadIdx.x; idx < WR * n_cta; idx += kThreads) {
        const int w_ = idx / n_cta, cl = idx - w_ * n_cta;
        const int rb = min((rowgroup * WR + w_) * 16, N - 1) / 128;
        bs_s[w_ * cpc + cl] = __ldg(p.w_s + static_cast<int64_t>(rb) * kc + c0 + cl);
    }
    __syncthreads();

    // ---- stream the weights
    float acc[MT][4];
#pragma unroll
    for (int j = 0; j < MT; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[j][i] = 0.0f;
    for (int i0 = 0; i0 < n_w; i0 += kRing) {
#pragma unroll
        for (int s = 0; s < kRing; ++s) {
            if (i0 + s < n_w) {
                const int c = w0 + i0 + s;
                const int cl = c - c0;
                const float bs = bs_s[wr * cpc + cl];
#pragma unroll
                for (int j = 0; j < MT; ++j) {
                    const uint8_t* xr = xq_s + (8 * j + g) * row_bytes + cl * kChunkK + 16 * t;
                    const uint4 f0 = *reinterpret_cast<const uint4*>(xr);
                    const uint4 f1 = *reinterpret_cast<const uint4*>(xr + 64);
                    float part[4];
                    chunk_product(part, ring[s], f0, f1);
                    // part[0..1]: weight row g, tokens 8j+2t, 8j+2t+1; part[2..3]: weight row g+8, same tokens
                    const float as0 = xs_s[(8 * j + 2 * t) * cpc + cl], as1 = xs_s[(8 * j + 2 * t + 1) * cpc + cl];
                    acc[j][0] = fmaf(part[0] * as0, bs, acc[j][0]);
                    acc[j][1] = fmaf(part[1] * as1, bs, acc[j][1]);
                    acc[j][2] = fmaf(part[2] * as0, bs, acc[j][2]);
                    acc[j][3] = fmaf(part[3] * as1, bs, acc[j][3]);
                }
                if (i0 + s + kRing < n_w) load_chunk(ring[s], c + kRing);
            }
        }
    }

    // ---- partial sums: the warps' meet in the CTA's shared memory, the CTAs' in that of the cluster's first one.  (Every
    // warp's 4-byte stores straight to the first CTA, tokens beyond M among them, made a launch up to 2.5 us slower: each is
    // a packet of its own, and one SM receives them all.)
#pragma unroll
    for (int j = 0; j < MT; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = g + ((i & 2) ? 8 : 0), tok = 8 * j + 2 * t + (i & 1);
            if (tok < p.M) slots[(wk * TOK + tok) * ROWS + wr * 16 + row] = acc[j][i];
        }
    __syncthreads();
    if (p.csize > 1) {
        cluster_wait();       // every CTA of the cluster runs
        const uint32_t first = mapa_shared(smem_u32(gathered), 0);
        for (int idx = threadIdx.x; idx < ROWS / 4 * p.M; idx += kThreads) {
            float4 sum = reinterpret_cast<const float4*>(slots)[idx];       // [token][rows]: idx runs over both
#pragma unroll
            for (int s = 1; s < WK; ++s) {
                const float4 v = reinterpret_cast<const float4*>(slots + s * TOK * ROWS)[idx];
                sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
            }
            st_cluster_f32x4(first + 4u * (rank * TOK * ROWS + 4 * idx), sum);
        }
        cluster_arrive();
        cluster_wait();
        if (rank != 0) return;
    }
    const float* src = p.csize > 1 ? gathered : slots;
    const int parts = p.csize > 1 ? p.csize : WK;
    for (int idx = threadIdx.x; idx < ROWS * p.M; idx += kThreads) {
        const int tok = idx / ROWS, rw = idx - tok * ROWS;
        const int n = rowgroup * ROWS + rw;
        if (n >= N) continue;
        float sum = 0.0f;
        for (int s = 0; s < parts; ++s) sum += src[s * TOK * ROWS + idx];
        p.c[static_cast<int64_t>(tok) * N + n] = __float2bfloat16_rn(sum);
    }
}

template <int WR, int WK, int MT, bool kFused>
int launch_variant(const SmallParams& prm, int rowgroups, size_t smem_bytes, cudaStream_t stream) {
    auto kern = fp8_linear_small_kernel<WR, WK, MT, kFused>;
    // the largest size there is, whatever this call needs: threads whose first calls differ set the same
    static bool configured[64] = {};
    int dev = 0;
    DSV3_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) {
        set_last_error("fp8_linear: device ordinal %d is outside the supported range", dev);
        return DSV3_ERR_UNSUPPORTED;
    }
    if (!configured[dev]) {
        DSV3_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kMaxSmem)));
        configured[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(rowgroups * prm.csize));
    cfg.blockDim = dim3(WR * WK * 32);
    cfg.dynamicSmemBytes = smem_bytes;
    cfg.stream = stream;
    // attributes: dependent launch first, the cluster dimension only when K is split over more than one CTA (a
    // cluster launch, even of one CTA, takes a slower path through the launch machinery)
    cudaLaunchAttribute attr[2];
    int n_attr = 0;
    if (pdl_enabled()) {
        attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n_attr].val.programmaticStreamSerializationAllowed = 1;
        ++n_attr;
    }
    if (prm.csize > 1) {
        attr[n_attr].id = cudaLaunchAttributeClusterDimension;
        attr[n_attr].val.clusterDim.x = static_cast<unsigned>(prm.csize);
        attr[n_attr].val.clusterDim.y = 1;
        attr[n_attr].val.clusterDim.z = 1;
        ++n_attr;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n_attr;
    DSV3_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, prm));
    return DSV3_OK;
}

}  // namespace

bool small_linear_supported(const void* act, const void* w, const void* c, int64_t M, int64_t N, int64_t K, bool fused) {
    const bool aligned = (reinterpret_cast<uintptr_t>(act) % 16) == 0 && (reinterpret_cast<uintptr_t>(w) % 16) == 0 &&
                         (reinterpret_cast<uintptr_t>(c) % 2) == 0;
    return aligned && M >= 1 && M <= 16 && N >= 1 && N < (1ll << 31) && K >= 16 && K < (1ll << 24) &&
           (K % (fused ? 128 : 16)) == 0;
}

// Automatic choice of the register-streaming kernel: up to 8 rows, up to 8 MB of weights in at most 4096 rows (its layout
// that splits K over the warps too).  It has less to set up than the tcgen05 pipeline; beyond 8 MB, or with more rows, the
// tcgen05 kernel's TMA ring streams as well or better.  B200, us, this kernel / tcgen05 at one row with weights from HBM: 1024 -> 2048 3.00 /
// 3.79; 7168 -> 576 4.00 / 4.89; 2048 -> 1408 3.07 / 4.11; 5120 -> 1536 4.88 / 5.36; 4096 -> 2048 4.21 / 5.31; 16384 -> 512 5.85 / 6.65; at eight
// rows 2048 -> 1408 3.07 / 4.31, 5120 -> 1536 4.89 / 5.52; beyond the line 7168 -> 1280 5.79 / 5.53, 7168 -> 1536 6.12 / 5.85, 4096 -> 3072 6.05 /
// 5.89, 5120 -> 3072 7.26 / 6.65; but 5120 -> 2048 4.96 / 5.66, 7168 -> 2048 6.18 / 6.45.  Within it, 71 to 73 row tiles of many chunks are more
// CTAs in clusters than there is room for: 7168 -> 1152 7.88 / 5.48.  K is bounded by the activations that a CTA stages, 128 K chunks even
// unsplit.
bool decode_kernel_pays(int64_t M, int64_t N, int64_t K) { return M <= 8 && N <= 4096 && K <= 16384 && N * K <= (8ll << 20); }

// x != nullptr: fused (bf16 activations); otherwise (a, a_s) are the quantised activations.
int launch_fp8_linear_small(const void* x, const void* a, const float* a_s, const void* w, const float* w_s, int64_t M,
                            int64_t N, int64_t K, int scale_fmt, void* c, cudaStream_t stream) {
    SmallParams prm;
    prm.x = static_cast<const uint4*>(x);
    prm.a = static_cast<const uint8_t*>(a);
    prm.a_s = a_s;
    prm.w = static_cast<const uint8_t*>(w);
    prm.w_s = w_s;
    prm.c = static_cast<__nv_bfloat16*>(c);
    prm.M = static_cast<int>(M);
    prm.N = static_cast<int>(N);
    prm.K = static_cast<int>(K);
    prm.kc = static_cast<int>((K + kChunkK - 1) / kChunkK);
    prm.scale_fmt = scale_fmt;
    // Layout: few weight rows -> a CTA takes one 16-row tile and its four (eight, sixteen) warps split K (more CTAs, and every CTA
    // quantises only its own K range); many rows -> a CTA takes four row tiles that share the staged activations.
    const bool narrow = N <= 4096;
    const int wr = narrow ? 1 : 4;
    int wk = narrow ? 4 : 1;
    const int rowgroups = static_cast<int>((N + 16 * wr - 1) / (16 * wr));
    // K splits across the CTAs of a cluster: enough CTAs for two per SM, at least 1.5 chunks per warp
    int csize = 1;
    while (csize < 8 && rowgroups * csize < 2 * num_sms() && prm.kc >= 3 * csize * wk) csize *= 2;
    // Up to 8 rows, half as many CTAs of eight warps instead, where that leaves no cluster to exchange sums in, or where clusters of
    // four-warp CTAs come near to filling the machine: registers admit four such CTAs per SM, 592, of which clusters of four and
    // eight find room for 568 (cudaOccupancyMaxActiveClusters); beyond, a second round costs as much as the first, and already
    // from 520 on the last clusters wait for room.  The line, three and a half per SM, is drawn by measurement.  us at 1 / 2 / 4
    // rows, four warps / eight: no cluster, 1536 -> 3072 4.1 / 4.6 / 4.7, 3.8 / 4.5 / 4.6, 2048 -> 2816 4.4 / 5.0 / 5.2, 4.1 / 4.8 / 5.0;
    // 7168 -> 2304 (576 CTAs) 10.5 / 10.9 / 13.0, 7.4 / 7.6 / 8.9; 7168 -> 2272 (568) 8.1 / 8.3 / 9.9, 7.4 / 7.5 / 8.8; 7168 -> 1040 (520 in
    // clusters of eight) 4.9 / 5.2 / 6.4, 4.8 / 5.2 / 5.4; but 5120 -> 2176 (544) 5.97 / 6.00 / 7.38, 6.00 / 6.05 / 7.53, 7168 -> 2048 (512)
    // 7.0 / 7.2 / 8.6, 7.15 / 7.3 / 8.7, 5120 -> 1536 (384) 5.5 / 5.6 / 6.9, 5.6 / 5.7 / 7.2; and at 16 rows, with twice the
    // accumulators, 1536 -> 3072 8.2, 12.6.  Each CTA then stages twice the K range: a K too long for that (beyond 24064
    // without a cluster) stays with four warps.
    const int mt = M <= 8 ? 1 : 2;
    const int tok = 8 * mt;
    auto smem_of = [&](int warps, int ctas) {
        const size_t cpc = static_cast<size_t>((prm.kc + ctas - 1) / ctas);
        return align16(static_cast<size_t>(tok) * (cpc * kChunkK + kRowPad)) + static_cast<size_t>(tok) * cpc * 4 +
               align16(static_cast<size_t>(wr) * cpc * 4) + static_cast<size_t>(ctas + warps) * wr * 16 * tok * 4 + 16;
    };
    // Where the row tiles are no more than the SMs and clusters would be of at most four, or no more than twice the SMs and no clusters
    // are needed, one CTA of sixteen or eight warps per row tile does without the exchange, and quantises the activations
    // with all of them (registers admit one such CTA per SM, or two).  us at 1 / 2 / 4 / 8 rows in a graph with weights from HBM, before / so: 2048 -> 1408
    // 3.69 / 4.07 / 4.21 / 5.33, 3.18 / 3.27 / 3.94 / 3.90; 1408 -> 2048 4.30 / 4.37 / 5.68 / 6.64, 2.97 / 3.02 / 3.59 / 3.46; 4096 -> 1536 4.40 /
    // 4.95 / 5.10 / 6.29, 4.18 / 4.75 / 4.98 / 6.17; 7168 -> 2048 6.78 / 6.93 / 8.08 / 10.67, 6.62 / 6.77 / 8.06 / 10.48; 7168 -> 2304 7.15 / 7.29 /
    // 8.47 / 10.82, 6.87 / 6.99 / 8.22 / 10.69; eight warps, 512 -> 4096 3.07 / 3.18 / 3.79 / 3.60, 2.66 / 2.72 / 2.77 / 3.13.  With more than 24
    // chunks to 80 to 127 row tiles the cluster is up to 3 % ahead in a graph, 7168 -> 1536 6.46 / 6.63 / 7.75, 6.62 / 6.69 / 7.95, 5120 -> 1536 5.34 /
    // 5.45 / 6.74, 5.40 / 5.46 / 6.87, 6144 -> 1280 5.72 / 5.79 / 7.11, 5.64 / 5.72 / 7.14, but behind where the launches come one by one, as a
    // cluster's launch takes longer: at 1 / 2 rows 6.95 / 7.10, 6.89 / 7.01; 6.05 / 6.11, 5.80 / 5.79; 6.38 / 6.47, 6.10 / 6.21 (weights in the
    // L2 6.38 / 6.57, 6.08 / 6.34; 5.53 / 5.62, 5.20 / 5.34; 5.82 / 5.91, 5.40 / 5.56).  Sixteen warps in
    // clusters of two instead of four in eight: 7168 -> 576 4.18 / 4.48 / 4.68, 4.32 / 4.99 / 5.25.  With activations that are quantised already only the exchange is gained, which few chunks, or few CTAs with many, do
    // not pay for: 1408 -> 2048 at one row 3.67, 2.92; but 256 -> 2048 2.47, 2.72; 1024 -> 1024 2.70, 2.82; 4096 -> 768 at eight rows 3.67,
    // 3.89.  (Both kinds of activations take the same layout: their results are the same bit for bit.)
    const bool pays = prm.kc >= 10 && (prm.kc <= 24 || rowgroups >= 80);
    if (narrow && M <= 8 && rowgroups <= num_sms() && csize <= 4 && pays && smem_of(16, 1) <= kMaxSmem) {
        wk = 16;
        csize = 1;
    } else if (narrow && M <= 8 && rowgroups <= 2 * num_sms() && rowgroups > num_sms() && csize == 1 && smem_of(8, 1) <= kMaxSmem) {
        wk = 8;
    } else if (narrow && M <= 8 && (csize == 2 || (csize > 2 && rowgroups * csize > 7 * num_sms() / 2)) && smem_of(8, csize / 2) <= kMaxSmem) {
        wk = 8;
        csize /= 2;
    }
    prm.csize = csize;
    prm.cpc = (prm.kc + csize - 1) / csize;
    const size_t smem = smem_of(wk, csize);
    if (smem > kMaxSmem) {
        set_last_error("fp8_linear: K=%lld is too long for the decode kernel's staging buffer", static_cast<long long>(K));
        return DSV3_ERR_UNSUPPORTED;
    }
    const bool fused = x != nullptr;
#define DSV3_SMALL_CASE(WR_, WK_, MT_, F_) return launch_variant<WR_, WK_, MT_, F_>(prm, rowgroups, smem, stream)
    if (wk == 16) {
        if (fused) DSV3_SMALL_CASE(1, 16, 1, true); else DSV3_SMALL_CASE(1, 16, 1, false);
    }
    if (wk == 8) {
        if (fused) DSV3_SMALL_CASE(1, 8, 1, true); else DSV3_SMALL_CASE(1, 8, 1, false);
    }
    if (narrow) {
        if (mt == 1) { if (fused) DSV3_SMALL_CASE(1, 4, 1, true); else DSV3_SMALL_CASE(1, 4, 1, false); }
        else         { if (fused) DSV3_SMALL_CASE(1, 4, 2, true); else DSV3_SMALL_CASE(1, 4, 2, false); }
    } else {
        if (mt == 1) { if (fused) DSV3_SMALL_CASE(4, 1, 1, true); else DSV3_SMALL_CASE(4, 1, 1, false); }
        else         { if (fused) DSV3_SMALL_CASE(4, 1, 2, true); else DSV3_SMALL_CASE(4, 1, 2, false); }
    }
#undef DSV3_SMALL_CASE
}

}  // namespace dsv3
