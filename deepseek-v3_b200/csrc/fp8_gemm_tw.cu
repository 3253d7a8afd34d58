// fp8_gemm for sm_100a, token-major tiles on CTA pairs with 256-wide accumulators: two CTAs (a cluster of two
// SMs) work on one 256 x 256 tile, each holding 128 token rows x 256 weight columns, with software promotion of
// every 128-wide K chunk.
//
// Replaces inference/kernel.py:118-172 (fp8_gemm_kernel) and its launch at :194-195 for prefill-sized M.
//
// Why 256 columns.  An SM takes about 60 bytes per clock from the L2: a chunk of 256 columns needs 32 KB of loads per SM for 512
// tensor-core cycles, one of 128 columns 24 KB for 256.  The price: the fp32 accumulator of one SM is 128 x 256 (128 registers in each
// of 256 promotion threads), TMEM holds only two chunk products, and the read-back buffer shrinks to 64 registers per thread.
//
// Why each product in two halves (N128).  A slot handed back as a whole was away for 1100 cycles besides its own 512 (commit, wake-up,
// two read-backs with the FMAs between them, arrivals from both CTAs, issue), so that two slots gave a product every 774 to 810 cycles.
// As halves, one for either warp group, the next product's left half is computed while the right one is still being read: 675.  The tokens
// are read from shared memory twice for that, 96 instead of 64 bytes per clock.  In a loop of launches the clock falls with the
// work it does (1 kW): us, whole slots / halves, act_quant included, M 500, N 7168, K 7168 35.6 / 34.2; M 867, N 18432, K 7168 126.8 / 123.4; M 4096, N 7168,
// K 16384 495 / 490; MLP 5120 -> 12288 at 2693 rows 538 / 521, 7168 -> 18432 at 8192 3098 / 3038.
//
// Roles, per CTA (r = rank in the pair; the even CTA is the leader):
//   warp 0            TMA producer (converged, one elected lane issues): stage = one K chunk = 16 KB tokens + 16 KB weights (64 rows
//                     of either 128-row block of the tile), five stages.  Both producers' loads complete on the LEADER's full[]
//                     barrier (ordinary, non-multicast loads; only the completion signal crosses to the peer),
//                     each waits on its own empty[].
//   warps 1,2         leader only: MMA issuers (converged, one elected lane issues); chunk g belongs to issuer g % 2, which owns TMEM slot g % 2.
//                     Per chunk: wait full[stage]; per half: wait tempty[half][slot] (8 arrivals: the half's promotion warps of both
//                     CTAs), 4 x tcgen05.mma.cta_group::2 kind::f8f6f4 (M256 N128 K32), commit -> tfull[half][slot] of both CTAs,
//                     behind the second half also empty[stage].  Stages alternate between the issuers, so full[] is waited for
//                     without a probe.
//   warps 4..11       promotion of this CTA's 128 x 256 half: warps 4..7 own columns 0..127 (one b_s block), warps
//                     8..11 columns 128..255; a thread owns one accumulator row.  A half product is read back in
//                     two pieces of 64 columns through one buffer; the half slot goes back to the issuer when the second
//                     load has landed, and that piece's FMAs follow the release.
//                     Result tile: bf16 through shared memory and TMA stores.
//
// One weight, or two of one size on the same activations (w1 and w3 of an MLP; TwOperands): a launch of 99 tiles on 74 pairs is two
// rounds, the second a third full, and two of them four; 198 tiles in one launch are three.  MLP 7168 -> 2304 at 2580 rows 158.8 / 144.1 us, 2048 -> 2816 at
// 3942 96.6 / 90.9, 5120 -> 12288 at 500 135.5 / 123.7, 2048 -> 1408 at 2580 45.6 / 41.5 (tw_two_pay()).  Tried instead: a launch each, the second
// one's CTAs on the SMs that the first one's last round leaves idle, without waiting for its end: 5 us more for the set-up of the CTAs (M 2580, N 2304,
// K 7168, w1 and w3 alone 120.9, in one launch 89.5, so 95.6), and nothing gained where more than half of the SMs have a tile in that round.
//
// Every mbarrier wait is bounded: after about a second the waiting thread records what it was waiting for in
// the status word, raises a CTA-wide abort flag and all roles fall through to the common teardown.  Before a
// CTA leaves, its producer waits for the last commits onto its empty[] barriers (nothing else would), and the
// pair meets at a cluster barrier, so that no signal is in flight towards a CTA that has gone.
#include <cuda.h>

#include <cstring>

#include "common.cuh"
#include "gemm_plan.cuh"
#include "tc_wait.cuh"

namespace dsv3 {

namespace {

constexpr int kNumThreads = 384;          // warp 0: TMA producer, warps 1-2: MMA issuers (leader), 3 idle, 4..11: promotion
constexpr int kFirstPromoWarp = 4;
constexpr int kPromoThreads = 256;
constexpr int kRegsControl = 40;
constexpr int kRegsPromo = 232;
// setmaxnreg.inc waits for registers of the CTA's pool, which is what the launch allocated (168 per thread, the
// most 384 threads can have): the two budgets must fit into it or the promotion warps would wait forever.
static_assert(128 * kRegsControl + 256 * kRegsPromo <= 384 * 168, "register pool");

constexpr int kBN = 256;                              // tile width: two b_s blocks, one per promotion warp group
constexpr int kBHalf = kBN / 2;                       // weight rows each CTA of the pair loads: half of either 128-row block
constexpr int kChunkBytes = (kPRows + kBHalf) * kChunk;   // per CTA: token tile + half weight tile of one chunk
constexpr int kStorePasses = 1;                       // result tile staged whole (1) or one 64-column box per warp group at a time (2)
constexpr int kStages = kStorePasses == 1 ? 5 : 6;    // of one chunk each
constexpr int kSlots = 2;                             // TMEM slots of one chunk product (two halves of 128 columns) each; barriers: [half][slot]
constexpr int kTmemCols = kSlots * kBN;
constexpr int kPiece = 32;                            // columns of an FMA batch; a read-back is two of them
constexpr int kStoreBytes = kPRows * kBN * 2 / kStorePasses;   // bf16 result tile: 128-byte-swizzled 128 x 64 boxes
constexpr int kSmemBytes = kStages * kChunkBytes + kStoreBytes + 1024 + 1024;
static_assert(kSmemBytes <= 232448, "shared memory per CTA");
static_assert(kSmemBytes > 116 * 1024, "one CTA per SM (it allocates all of TMEM)");
static_assert(kTmemCols == 512, "all of TMEM");
// The issuers alternate, so a stage's full[] barrier is waited for by one issuer at one use and by the other at the
// next.  A parity wait is only exact for a barrier that is at most one phase behind.  That holds here: an issuer
// reaches chunk g after it was given both halves of its TMEM slot for chunk g - 2, i.e. after the promotion warps have read chunk
// g - 4 and, in order, every chunk before it -- among them chunk g - kStages, the stage's previous use, whose
// product could only exist after the other issuer had waited for that use's loads.
static_assert(kStages >= 4 && kSlots == 2, "phase argument for the full[] waits of alternating issuers");
static_assert((kPRows * kChunk) % 1024 == 0 && kChunkBytes % 1024 == 0, "operand tiles keep the swizzle atom's alignment");

struct TwParams {
    const float* a_s;
    const float* b_s;
    __nv_bfloat16* c;
    unsigned int* status;
    int64_t M, N;
    int kc;                 // K chunks
    int nblk;               // rows of b_s (128-wide weight blocks)
    int tiles_pp, tiles_q;  // pairs of token tiles, 256-wide weight tiles
    int raster;             // token-tile pairs that share consecutive weight tiles in the work order
    FastDiv div_per_group, div_raster;
    int tma_store;          // results leave through shared memory and a TMA store (needs N % 8 == 0)
    int num_tiles;          // whole tiles: all, or all but those of the last round
    int tail_tiles, tail_w; // tiles shared out in strips of tail_w columns (128 or 64) instead, one strip per pair; 0: none
};

// Operands as tensor maps.  Two weights (w1 and w3 of an MLP, equal in size, on the same activations): the second one's tiles follow
// the first one's in the order of weight tiles, so that the two have one last round between them.
template <int kMats>
struct TwOperands;
template <>
struct TwOperands<1> {
    CUtensorMap a, b[1], c[1], s[1];      // s: strips' boxes of b
};
template <>
struct TwOperands<2> {
    CUtensorMap a, b[2], c[2], s[2];
    const float* b_s1;                    // the second weight's, beside TwParams::b_s and c
    __nv_bfloat16* c1;
    int tiles_q0;                         // weight tiles of the first
};

struct Tile {
    int pp, q;
    int m;                  // which weight
};

template <int kMats>
__device__ __forceinline__ const float* b_s_of(const TwOperands<kMats>& o, const TwParams& p, int m) {
    if constexpr (kMats == 2) {
        if (m) return o.b_s1;
    }
    return p.b_s;
}
template <int kMats>
__device__ __forceinline__ __nv_bfloat16* c_of(const TwOperands<kMats>& o, const TwParams& p, int m) {
    if constexpr (kMats == 2) {
        if (m) return o.c1;
    }
    return p.c;
}

// Work order: `raster` token-tile pairs share consecutive weight tiles so that a wave re-uses both operands in L2.
template <int kMats>
__device__ __forceinline__ Tile decode_tile(int tile, const TwOperands<kMats>& o, const TwParams& p) {
    const int per_group = p.raster * p.tiles_q;
    const int grp = static_cast<int>(fast_div(static_cast<uint32_t>(tile), p.div_per_group));
    const int first = grp * p.raster;
    const int gsz = min(p.raster, p.tiles_pp - first);
    const int r = tile - grp * per_group;
    Tile t;
    t.q = (gsz == p.raster) ? static_cast<int>(fast_div(static_cast<uint32_t>(r), p.div_raster)) : r / gsz;   // the last group may be shorter
    t.pp = first + (r - t.q * gsz);
    t.m = 0;
    if constexpr (kMats == 2) {
        if (t.q >= o.tiles_q0) {
            t.q -= o.tiles_q0;
            t.m = 1;
        }
    }
    return t;
}

// The last round.  A machine of 74 pairs works on 448 tiles in six rounds and a seventh of four tiles, which takes as long as the
// others while 70 pairs have nothing to do.  Where at most half of the pairs would have a tile in the last round, its
// tiles are cut into strips of 128 or 64 columns, one per pair: a strip loads its tokens like a tile but multiplies a half or a
// quarter of it, and needs no exchange with the others (every column is summed in the same order: the result is the same bit
// for bit).  A chunk then takes 0.37 or 0.27 us (the loads in flight) instead of 0.41.  B200, us, whole tiles / strips: M 4096,
// N 7168, K 16384 (448 tiles) 476 / 460; M 8192, N 7168, K 18432 (896) 1048 / 1024; M 8192, N 18432, K 7168 (2304) 988 / 979;
// M 1003, N 576, K 7168 (12) 25.1 / 18.8.
struct Strip {
    Tile t;
    int n0;                 // first column
    bool any;
};
template <int kMats>
__device__ __forceinline__ Strip decode_strip(int pair, const TwOperands<kMats>& o, const TwParams& p) {
    Strip s = {};
    const int shift = p.tail_w == 64 ? 2 : 1;
    if (p.tail_w == 0 || (pair >> shift) >= p.tail_tiles) return s;
    s.t = decode_tile(p.num_tiles + (pair >> shift), o, p);
    s.n0 = s.t.q * kBN + (pair & ((1 << shift) - 1)) * p.tail_w;
    s.any = s.n0 < p.N;
    return s;
}

// kBlock: K chunks per scale load: 4 (K chunks a multiple of four, 16-byte aligned scales), 2 (of two, 8-byte), else 1, or kShifted: in the
// aligned groups of four that rows lie in, wherever they begin
constexpr int kShifted = 0, kShiftedFrom = 19;
template <int kBlock, int kMats>
__global__ void __launch_bounds__(kNumThreads, 1)
fp8_gemm_tw_kernel(const __grid_constant__ TwOperands<kMats> o, const TwParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t tiles = (raw + 1023u) & ~1023u;     // the same offset in both CTAs of the pair
    uint8_t* gen_tiles = smem_raw + (tiles - raw);
    uint8_t* store_buf = gen_tiles + kStages * kChunkBytes;                       // 1024-byte aligned (swizzle atom)
    uint64_t* bars = reinterpret_cast<uint64_t*>(store_buf + kStoreBytes);
    Control* ctl = reinterpret_cast<Control*>(bars + 2 * kStages + 4 * kSlots);
    const uint32_t bar0 = smem_u32(bars);
    auto full_bar = [&](int s) { return bar0 + 8u * s; };                        // used in the leader only
    auto empty_bar = [&](int s) { return bar0 + 8u * (kStages + s); };
    auto tfull_bar = [&](int s) { return bar0 + 8u * (2 * kStages + s); };
    auto tempty_bar = [&](int s) { return bar0 + 8u * (2 * kStages + 2 * kSlots + s); };   // used in the leader only

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);   // uniform, and known to be
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();            // 0: leader (issues the MMAs), 1: peer
    const int pair = static_cast<int>(blockIdx.x >> 1);
    const int n_pairs = static_cast<int>(gridDim.x >> 1);
    const int kc = p.kc;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int s = 0; s < 2 * kSlots; ++s) {
            mbar_init(tfull_bar(s), 1);
            mbar_init(tempty_bar(s), kPromoThreads / 32);       // one warp group of each CTA reads a half
        }
        ctl->abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&o.a);
        for (int m = 0; m < kMats; ++m) {
            tma_prefetch_desc(&o.b[m]);
            if (p.tma_store) tma_prefetch_desc(&o.c[m]);
        }
    }
    if (warp == 1) tc_alloc_pair(smem_u32(&ctl->tmem_base), kTmemCols);
    // Programmatic dependent launch: nothing above touches global memory, so it may overlap the tail of
    // the kernel before this one in the stream.  While waiting for that kernel, the producer thread pulls
    // the first weight boxes of this CTA's first tile into L2 (L2 is the point of coherence: should the
    // predecessor still be writing those weights, the later TMA loads see its data all the same).
    if (threadIdx.x == 0) {
        const int n_pre = min(kc, kStages);
        if (pair < p.num_tiles) {
            const Tile t = decode_tile(pair, o, p);
            for (int j = 0; j < n_pre; ++j)
                for (int h = 0; h < 2; ++h) tma_prefetch_l2_2d(&o.b[t.m], j * kChunk, t.q * kBN + h * kBHalf + static_cast<int>(rank) * (kBHalf / 2));
        } else if (const Strip s = decode_strip(pair, o, p); s.any) {
            for (int j = 0; j < n_pre; ++j) tma_prefetch_l2_2d(&o.s[s.t.m], j * kChunk, s.n0 + static_cast<int>(rank) * (p.tail_w / 2));
        }
    }
    griddep_launch_dependents();
    // the peer's barriers must be initialised before anything is signalled across the pair
    tc_fence_before();
    __syncthreads();
    cluster_arrive();
    cluster_wait();
    tc_fence_after();
    griddep_wait();
    const uint32_t tmem_base = ctl->tmem_base;

    if (warp < kFirstPromoWarp) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsControl));
        if (warp == 0) {
            // ------------------------------------------------------------ TMA producer (both CTAs)
            // (converged warp, elected lane: see the issuers)
            {
                uint32_t g = 0;
                uint32_t probe = 0;   // result of test_wait on empty[] for chunk g, issued one chunk earlier
                bool ok = true;
                auto load_tile = [&](const void* tmap, int boxes, int a_row, int b_row, uint32_t bytes) {
                    for (int k = 0; k < kc; ++k, ++g) {
                        const int s = g % kStages;
                        ok = __all_sync(0xffffffffu, wait_probed(probe, empty_bar(s), ((g / kStages) & 1u) ^ 1u, ctl, p.status, 1, g));
                        if (!ok) break;
                        probe = mbar_test_wait(empty_bar((g + 1) % kStages), (((g + 1) / kStages) & 1u) ^ 1u) ? 1u : 0u;
                        const uint32_t lead_full = mapa_shared(full_bar(s), 0);
                        // the leader's barrier expects the bytes of both CTAs; the peer's loads may complete on it
                        // before this arrive has been made (the phase cannot complete without it)
                        const uint32_t dst = tiles + s * kChunkBytes;
                        if (elect_one()) {
                            if (rank == 0) mbar_arrive_expect_tx(full_bar(s), bytes);
                            tma_load_2d_pair(dst, &o.a, k * kChunk, a_row, lead_full);
                            tma_load_2d_pair(dst + kPRows * kChunk, tmap, k * kChunk, b_row, lead_full);
                            if (boxes == 2) tma_load_2d_pair(dst + kPRows * kChunk + kBHalf / 2 * kChunk, tmap, k * kChunk, b_row + kBHalf, lead_full);
                        }
                        __syncwarp();
                    }
                };
                for (int tile = pair; ok && tile < p.num_tiles; tile += n_pairs) {
                    const Tile t = decode_tile(tile, o, p);
                    load_tile(&o.b[t.m], 2, (2 * t.pp + static_cast<int>(rank)) * kPRows, t.q * kBN + static_cast<int>(rank) * (kBHalf / 2), 2 * kChunkBytes);
                }
                if (const Strip st = decode_strip(pair, o, p); ok && st.any)
                    load_tile(&o.s[st.t.m], 1, (2 * st.t.pp + static_cast<int>(rank)) * kPRows, st.n0 + static_cast<int>(rank) * (p.tail_w / 2),
                              2u * (kPRows + p.tail_w / 2) * kChunk);
                // Nothing waits for the commits onto the empty[] barriers of the last chunks; wait for them here so
                // that none is in flight when the CTA leaves (it would land in whatever CTA gets this shared memory next).
                for (uint32_t d = (g > kStages ? g - kStages : 0u); ok && d < g; ++d)
                    ok = __all_sync(0xffffffffu, bounded_wait(empty_bar(d % kStages), (d / kStages) & 1u, ctl, p.status, 1, d));
            }
        } else if (warp <= 2) {
            // ------------------------------------------------------------ MMA issuers (leader CTA; chunk g -> issuer g % 2)
            // One thread issues about one tcgen05 instruction per hundred cycles, and a chunk costs fourteen (eight MMAs,
            // six commits) for 512 tensor-core cycles: two threads share the chunks, each owning one TMEM slot.
            // The whole warp walks the loop (waits included) and one elected lane issues: control flow, addresses
            // and descriptors then stay warp-uniform, which is what makes a tcgen05 instruction cheap to issue.
            if (rank == 0) {
                const uint32_t me = static_cast<uint32_t>(warp - 1);
                const int slot = static_cast<int>(me);
                const uint32_t peer_tfull0 = mapa_shared(tfull_bar(0), 1);
                const uint32_t peer_empty0 = mapa_shared(empty_bar(0), 1);
                const uint32_t d_tmem = tmem_base + slot * kBN;
                bool ok = true;
                uint32_t g = 0;
                // parts == 2: the halves of a tile, one after the other; 1: a strip, which both warp groups read
                auto multiply_tile = [&](uint32_t idesc, int parts) {
                    for (int k = 0; k < kc; ++k, ++g) {
                        if ((g & 1u) != me) continue;
                        const int s = g % kStages;
                        ok = __all_sync(0xffffffffu, bounded_wait(full_bar(s), (g / kStages) & 1u, ctl, p.status, 2, g));
                        if (!ok) break;
                        const uint32_t sp = tiles + s * kChunkBytes;
                        const uint64_t da = umma_desc_k_major_sw128(sp);
                        for (int h = 0; h < parts; ++h) {
                            ok = __all_sync(0xffffffffu, bounded_wait(tempty_bar(h * kSlots + slot), ((g >> 1) & 1u) ^ 1u, ctl, p.status, 3, g) &&
                                                         (parts == 2 || bounded_wait(tempty_bar(kSlots + slot), ((g >> 1) & 1u) ^ 1u, ctl, p.status, 3, g)));
                            if (!ok) break;
                            tc_fence_after();
                            const uint64_t db = umma_desc_k_major_sw128(sp + kPRows * kChunk + h * (kBHalf / 2) * kChunk);
                            if (elect_one()) {
#pragma unroll
                                for (int kk = 0; kk < kChunk / 32; ++kk) {
                                    // 32 bytes further along K inside the 128-byte swizzle atom: +2 in address units of 16 B
                                    tc_mma_f8_pair(d_tmem + h * kBHalf, da + 2u * kk, db + 2u * kk, idesc, kk > 0 ? 1u : 0u);
                                }
                                // this product is complete in the TMEM of both CTAs; behind the last one the stage is reusable in both
                                tc_commit_pair(tfull_bar(h * kSlots + slot));
                                tc_commit_pair(peer_tfull0 + 8u * (h * kSlots + slot));
                                if (parts == 1) {
                                    tc_commit_pair(tfull_bar(kSlots + slot));
                                    tc_commit_pair(peer_tfull0 + 8u * (kSlots + slot));
                                }
                                if (h == parts - 1) {
                                    tc_commit_pair(empty_bar(s));
                                    tc_commit_pair(peer_empty0 + 8u * s);
                                }
                            }
                            __syncwarp();
                        }
                        if (!ok) break;
                    }
                };
                for (int tile = pair; ok && tile < p.num_tiles; tile += n_pairs) multiply_tile(umma_idesc_e4m3_f32(2 * kPRows, kBHalf), 2);
                if (ok && decode_strip(pair, o, p).any) multiply_tile(umma_idesc_e4m3_f32(2 * kPRows, static_cast<uint32_t>(p.tail_w)), 1);
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsPromo));
        // ------------------------------------------------------------ promotion + epilogue (both CTAs)
        // Warps 4..7 own the left 128 columns of the CTA's 128 x 256 half, warps 8..11 the right 128; within a
        // column half a thread owns one accumulator row (TMEM lane).
        const int half = (warp - kFirstPromoWarp) >> 2;
        const int col0 = half * 128;
        const int quarter = warp & 3;                       // TMEM lane quarter this warp may access
        const int row = quarter * 32 + lane;                // accumulator row (TMEM lane)
        const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + col0;
        const uint32_t lead_tempty0 = mapa_shared(tempty_bar(half * kSlots), 0);   // this group's first, in the leader

        uint32_t v[2][kPiece];
        float2 acc[64];
        // fold piece `pc` of a chunk product (a constant once the loops around the calls are unrolled)
        auto fold = [&](const uint32_t* vv, float sc, int pc) {
            const float2 sc2 = make_float2(sc, sc);
#pragma unroll
            for (int j = 0; j < kPiece / 2; ++j)
                acc[pc * (kPiece / 2) + j] = __ffma2_rn(make_float2(__uint_as_float(vv[2 * j]), __uint_as_float(vv[2 * j + 1])), sc2,
                                                        acc[pc * (kPiece / 2) + j]);
        };
        auto release = [&](int slot) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(lead_tempty0 + 8u * slot);
        };
        // Result tile: the four warps of a column half stage their two 128 x 64 bf16 boxes in shared memory (128-byte
        // swizzle: 16-byte slot c of row r sits at slot c ^ (r & 7), which also keeps the vector stores free of
        // bank conflicts) and one thread hands them to the TMA, which clips rows beyond M and columns beyond N.
        // The stores of the previous tile are only known to have read the buffer once their issuer has waited for
        // them, hence the first barrier, which every tile passes and which also says whether a wait of any of the four
        // warps gave up (false: they all turn away).  tp = token tile of this CTA.
        const bool issuer = (((threadIdx.x - kFirstPromoWarp * 32) & 127) == 0);
        auto write_tile = [&](int tp, int tq, int m) -> bool {
            if (p.tma_store) {
                if (issuer) bulk_wait_group_read0();
                if (!barrier_all<128>(2 + half, true)) return false;
            }
            if (static_cast<int64_t>(tp) * kPRows >= p.M) return true;     // the odd half of the last pair: nothing to store
            const int64_t n0 = static_cast<int64_t>(tq) * kBN + col0;
            if (n0 >= p.N) return true;                                    // the tile's right half lies beyond N
            if (p.tma_store) {
                constexpr int kBoxes = 2 / kStorePasses;               // boxes per warp group and pass
                uint8_t* sbuf = store_buf + half * (kBoxes * kPRows * 128);
#pragma unroll
                for (int pass = 0; pass < kStorePasses; ++pass) {
                    if (pass > 0) {
                        if (issuer) bulk_wait_group_read0();
                        asm volatile("bar.sync %0, 128;" ::"r"(2 + half) : "memory");
                    }
#pragma unroll
                    for (int c8 = 0; c8 < 8 * kBoxes; ++c8) {      // 16-byte slot of the thread's columns: box cc / 8, slot cc % 8
                        const int cc = pass * 8 * kBoxes + c8;
                        const uint4 o = make_uint4(pack_bf16x2(acc[4 * cc].x, acc[4 * cc].y), pack_bf16x2(acc[4 * cc + 1].x, acc[4 * cc + 1].y),
                                                   pack_bf16x2(acc[4 * cc + 2].x, acc[4 * cc + 2].y), pack_bf16x2(acc[4 * cc + 3].x, acc[4 * cc + 3].y));
                        *reinterpret_cast<uint4*>(sbuf + (c8 >> 3) * (kPRows * 128) + row * 128 + (((c8 & 7) ^ (row & 7)) << 4)) = o;
                    }
                    fence_proxy_async_shared();
                    asm volatile("bar.sync %0, 128;" ::"r"(2 + half) : "memory");
                    if (issuer) {
#pragma unroll
                        for (int bx = 0; bx < kBoxes; ++bx) {
                            const int64_t n = n0 + (pass * kBoxes + bx) * 64;
                            if (n < p.N) tma_store_2d(&o.c[m], smem_u32(sbuf + bx * (kPRows * 128)), static_cast<int>(n), tp * kPRows);
                        }
                        bulk_commit_group();
                    }
                }
            } else {
                const int64_t tok = static_cast<int64_t>(tp) * kPRows + row;
                const int64_t N = p.N;
                if (tok < p.M) {
                    __nv_bfloat16* crow = c_of(o, p, m) + tok * N;
#pragma unroll
                    for (int j = 0; j < 64; ++j) {
                        if (n0 + 2 * j < N) crow[n0 + 2 * j] = __float2bfloat16_rn(acc[j].x);
                        if (n0 + 2 * j + 1 < N) crow[n0 + 2 * j + 1] = __float2bfloat16_rn(acc[j].y);
                    }
                }
            }
            return true;
        };

        // Scale rows of a tile for this thread, as element offsets: a_s of its token (clamped at the edge), b_s of
        // the weight block of its column half (clamped where that half lies beyond N).
        auto as_row = [&](const Tile& t) {
            const int64_t tok = static_cast<int64_t>(2 * t.pp + static_cast<int>(rank)) * kPRows + row;
            return p.a_s + min(tok, p.M - 1) * kc;
        };
        auto bs_row = [&](const Tile& t) { return b_s_of(o, p, t.m) + static_cast<int64_t>(min(2 * t.q + half, p.nblk - 1)) * kc; };

        // Scales, kBlock chunks at a time.  A thread's a_s row is a 32-byte sector of its own, and L1 (what the operand
        // stages leave of it) does not hold 256 of them until the next chunk: one chunk at a time, the scales cost a quarter
        // as much L2 traffic as the operands and a wait in every chunk (M 4096, N 7168, K 16384: 465 us, with no scale loads
        // at all 419, as here 430; with products in halves 394, with no loads 367, eight chunks at a time 458).  One 16-byte load brings
        // four chunks; it is issued as soon as the fourth product is formed and has that chunk's time to arrive.  Rows that 16-byte loads cannot read (K chunks not a
        // multiple of four) take 8-byte loads, kBlock = 2, or others; scalar / 8-byte, M 4096, N 7168, K 2304 64.2 / 62.6 us, M 8862,
        // N 2608, K 8960 195.4 / 190.7, M 2000, N 2048, K 2816 15.9 / 15.5.
        // From kShiftedFrom chunks rows that begin anywhere are read in aligned groups of four, too, two of which hold the next four chunks: a
        // thread picks them out by its own row's offset, and the last one to three chunks come behind the groups of four.  A scalar load waits in every
        // chunk, which products in halves had made longer than what it was before them.  us with act_quant, whole slots and scalar loads / halves and scalar / so: M 2456, N 5456,
        // K 6272 102.9 / 104.6 / 97.7; M 4096, N 7168, K 7296 247.1 / 251.1 / 236.8; M 8192, N 5120, K 12416 631 / 630 / 551.  Shorter rows are over before it pays: with
        // 3 to 9 chunks 1 to 5 % slower, with 11, 13, 15 and 17 level, 1 to 2 % slower, 1 % faster and level, with 19 1 to 3 % faster.  (Even numbers of chunks: 4 to 6 % slower than 8-byte loads.)
        float ra[kBlock == kShifted ? 1 : kBlock], rb[kBlock == kShifted ? 4 : kBlock];
        float4 a_cur, a_next;      // kShifted: the groups that hold the next four chunks' a_s
        const float* const a_end = p.a_s + p.M * kc;
        // group `grp` of a row; nothing outside of a_s is read
        const auto offset_of = [](const float* row) { return static_cast<int>((reinterpret_cast<uintptr_t>(row) >> 2) & 3); };
        auto a_group = [&](const float* row, int grp) -> float4 {
            // (predicated, not branched around: behind a branch a load is waited for at once)
            const float* q = row - offset_of(row) + 4 * grp;
            const bool whole = q >= p.a_s && q + 4 <= a_end;
            float4 e = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const auto one = [&](float& x, int i) {
                asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %1, 0;\n @p ld.global.nc.f32 %0, [%2];\n}"
                             : "+f"(x) : "r"(static_cast<int>(!whole && q + i >= p.a_s && q + i < a_end)), "l"(q + i));
            };
            asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n @p ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%5];\n}"
                         : "+f"(e.x), "+f"(e.y), "+f"(e.z), "+f"(e.w) : "r"(static_cast<int>(whole)), "l"(q));
            one(e.x, 0);
            one(e.y, 1);
            one(e.z, 2);
            one(e.w, 3);
            return e;
        };
        auto next_scales = [&](const float* as, const float* bs, int k) {
            if (k >= kc) return;
            if constexpr (kBlock == 4) {
                const float4 a4 = __ldg(reinterpret_cast<const float4*>(as + k)), b4 = __ldg(reinterpret_cast<const float4*>(bs + k));
                ra[0] = a4.x; ra[1] = a4.y; ra[2] = a4.z; ra[3] = a4.w;
                rb[0] = b4.x; rb[1] = b4.y; rb[2] = b4.z; rb[3] = b4.w;
            } else if constexpr (kBlock == 2) {
                const float2 a2 = __ldg(reinterpret_cast<const float2*>(as + k)), b2 = __ldg(reinterpret_cast<const float2*>(bs + k));
                ra[0] = a2.x; ra[1] = a2.y;
                rb[0] = b2.x; rb[1] = b2.y;
            } else if constexpr (kBlock == 1) {
                ra[0] = __ldg(as + k);
                rb[0] = __ldg(bs + k);
            } else {
                a_cur = k == 0 ? a_group(as, 0) : a_next;
                a_next = a_group(as, k / 4 + 1);
#pragma unroll
                for (int i = 0; i < 4; ++i) rb[i] = __ldg(bs + min(k + i, kc - 1));
            }
        };
        // kShifted: the products of the four
        auto take_scales = [&](const float* as, float (&sc)[4]) {
            const int m = offset_of(as);
            const bool one = m & 1, two = m & 2;
            const float t0 = one ? a_cur.y : a_cur.x, t1 = one ? a_cur.z : a_cur.y, t2 = one ? a_cur.w : a_cur.z;
            const float t3 = one ? a_next.x : a_cur.w, t4 = one ? a_next.y : a_next.x, t5 = one ? a_next.z : a_next.y;
            sc[0] = (two ? t2 : t0) * rb[0];
            sc[1] = (two ? t3 : t1) * rb[1];
            sc[2] = (two ? t4 : t2) * rb[2];
            sc[3] = (two ? t5 : t3) * rb[3];
        };
        auto first_scales = [&](const Tile& t) { next_scales(as_row(t), bs_row(t), 0); };
        bool ok = true;
        uint32_t g = 0;            // chunk counter
        int tile = pair;
        if (tile < p.num_tiles) {
            Tile cur = decode_tile(tile, o, p);
            first_scales(cur);
            while (true) {
                const float* as_ptr = as_row(cur);
                const float* bs_ptr = bs_row(cur);
#pragma unroll
                for (int j = 0; j < 64; ++j) acc[j] = make_float2(0.0f, 0.0f);
                // one chunk; scale(): its scale, formed (and the next ones asked for) while its first columns are on their way
                auto chunk = [&](auto scale) {
                    const int slot = static_cast<int>(g & 1u);
                    const bool mine = bounded_wait_lean(tfull_bar(half * kSlots + slot), (g >> 1) & 1u, ctl, p.status, 4, g);
                    ++g;
                    ok = __all_sync(0xffffffffu, mine);
                    if (!ok) return;
                    tc_fence_after();
                    const uint32_t t_slot = t_lane + slot * kBN;
                    // The first 64 columns are read back and folded, then the other 64 are read back and the half slot
                    // returns to the issuer: two read-back latencies per chunk; the last fold follows the release.
                    tc_ld_x64(t_slot, &v[0][0]);
                    const float sc = scale();
                    tc_wait_ld();
                    fold(v[0], sc, 0);
                    fold(v[1], sc, 1);
                    tc_ld_x64(t_slot + 2 * kPiece, &v[0][0]);
                    tc_wait_ld();
                    release(slot);
                    fold(v[0], sc, 2);
                    fold(v[1], sc, 3);
                };
                if constexpr (kBlock == kShifted) {
                    int k0 = 0;
                    float sc[4];
                    for (; ok && k0 + 4 <= kc; k0 += 4) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            chunk([&] {
                                if (i == 0) take_scales(as_ptr, sc);
                                if (i == 3) next_scales(as_ptr, bs_ptr, k0 + 4);
                                return sc[i];
                            });
                            if (!ok) break;
                        }
                    }
                    for (int i = 0; ok && i < kc - k0; ++i)
                        chunk([&] {
                            if (i == 0) take_scales(as_ptr, sc);
                            return i == 0 ? sc[0] : (i == 1 ? sc[1] : sc[2]);
                        });
                } else {
                    for (int k0 = 0; ok && k0 < kc; k0 += kBlock) {
#pragma unroll
                        for (int i = 0; i < kBlock; ++i) {
                            chunk([&] {
                                const float sc = ra[i] * rb[i];
                                if (i == kBlock - 1) next_scales(as_ptr, bs_ptr, k0 + kBlock);
                                return sc;
                            });
                            if (!ok) break;
                        }
                    }
                }
                if (!ok) {
                    if (p.tma_store) barrier_all<128>(2 + half, false);
                    break;
                }
                // the next tile's first scales are requested before this tile is written, so that their latency
                // (and the tile decode) hides under the epilogue while the issuer already fills both TMEM slots
                const int next = tile + n_pairs;
                const bool more = next < p.num_tiles;
                Tile nt = cur;
                if (more) {
                    nt = decode_tile(next, o, p);
                    first_scales(nt);
                }
                ok = write_tile(2 * cur.pp + static_cast<int>(rank), cur.q, cur.m);
                if (!ok || !more) break;
                tile = next;
                cur = nt;
            }
        }
        // ---- a strip of the last round: the two warp groups take half of its columns each, and store them directly
        if (const Strip st = decode_strip(pair, o, p); ok && st.any) {
            const int cw = p.tail_w / 2, n0 = st.n0 + half * cw;
            const float* as_ptr = as_row(st.t);
            const float* bs_ptr = b_s_of(o, p, st.t.m) + static_cast<int64_t>(st.n0 / 128) * kc;
            // scales are requested four chunks ahead: a chunk takes half as long as a load that misses L1
            float sa[4], sb[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                sa[i] = __ldg(as_ptr + min(i, kc - 1));
                sb[i] = __ldg(bs_ptr + min(i, kc - 1));
            }
#pragma unroll
            for (int j = 0; j < 32; ++j) acc[j] = make_float2(0.0f, 0.0f);
            const uint32_t t_strip = t_lane - col0 + half * cw;
            for (int k0 = 0; ok && k0 < kc; k0 += 4) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (k0 + i >= kc) break;
                    const int slot = static_cast<int>(g & 1u);
                    ok = __all_sync(0xffffffffu, bounded_wait_lean(tfull_bar(half * kSlots + slot), (g >> 1) & 1u, ctl, p.status, 4, g));
                    ++g;
                    if (!ok) break;
                    tc_fence_after();
                    const float sc = sa[i] * sb[i];
                    if (cw == 64) tc_ld_x64(t_strip + slot * kBN, &v[0][0]);
                    else tc_ld_x32(t_strip + slot * kBN, &v[0][0]);
                    sa[i] = __ldg(as_ptr + min(k0 + i + 4, kc - 1));
                    sb[i] = __ldg(bs_ptr + min(k0 + i + 4, kc - 1));
                    tc_wait_ld();
                    release(slot);
                    fold(v[0], sc, 0);
                    if (cw == 64) fold(v[1], sc, 1);
                }
            }
            const int64_t m = static_cast<int64_t>(2 * st.t.pp + static_cast<int>(rank)) * kPRows + row;
            if (ok && m < p.M) {
                __nv_bfloat16* crow = c_of(o, p, st.t.m) + m * p.N;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int n = n0 + 8 * j;
                    if (8 * j >= cw || n >= p.N) break;
                    if (p.tma_store) {                              // (N % 8 == 0)
                        *reinterpret_cast<uint4*>(crow + n) = make_uint4(pack_bf16x2(acc[4 * j].x, acc[4 * j].y), pack_bf16x2(acc[4 * j + 1].x, acc[4 * j + 1].y),
                                                                         pack_bf16x2(acc[4 * j + 2].x, acc[4 * j + 2].y), pack_bf16x2(acc[4 * j + 3].x, acc[4 * j + 3].y));
                    } else {
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            if (n + e < p.N) crow[n + e] = __float2bfloat16_rn(e & 1 ? acc[4 * j + e / 2].y : acc[4 * j + e / 2].x);
                    }
                }
            }
        }
    }

    // ---------------------------------------------------------------- teardown
    if (warp >= kFirstPromoWarp && ((threadIdx.x - kFirstPromoWarp * 32) & 127) == 0) bulk_wait_group0();   // result tiles have left shared memory
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (ctl->abort_flag) {
        // give copies and MMAs that were already issued time to land before the CTA's
        // shared memory and TMEM are released
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
        __syncthreads();
    }
    // neither CTA of the pair may go while the other can still signal its barriers or read its operands
    cluster_arrive();
    cluster_wait();
    if (warp == 1) {
        tc_fence_after();
        tc_dealloc_pair(tmem_base, kTmemCols);
    }
}

}  // namespace

bool tw_pair_supported(int64_t M, int64_t N, int64_t K) {
    (void)K;
    // At least two token tiles (otherwise the second CTA of a pair would multiply zeros) and more than one weight
    // block (otherwise half of every accumulator would).  Whether it is the faster kernel for a problem is the
    // plan's decision (tc_plan).
    return M > kPRows && N > 128;
}

// (128-wide strips of a short K gain nothing: M 2063, N 7168, K 2304, 30 of 252 tiles, 37.9 us whole, 38.5 in strips)
int tw_strip_width(int64_t tiles, int64_t pairs, int kc) {
    if (tiles == 0 || 2 * tiles > pairs) return 0;
    return 4 * tiles <= pairs ? 64 : (kc >= 24 ? 128 : 0);
}

namespace {

template <int kMats>
int launch(const void* a, const float* a_s, const void* const* b, const float* const* b_s, int64_t M, int64_t N, int64_t K, void* const* c,
           cudaStream_t stream) {
    const int64_t tiles_p = (M + kPRows - 1) / kPRows, tiles_q0 = (N + kBN - 1) / kBN;
    const int64_t tiles_pp = (tiles_p + 1) / 2, tiles_q = kMats * tiles_q0;
    if (tiles_pp * tiles_q >= (1ll << 31)) {
        set_last_error("fp8_gemm: %lld x %lld output tiles are more than the work-item counter holds",
                       static_cast<long long>(tiles_p), static_cast<long long>(tiles_q));
        return DSV3_ERR_UNSUPPORTED;
    }
    TwOperands<kMats> ops;
    memset(&ops, 0, sizeof(ops));
    int rc;
    if ((rc = make_tmap(&ops.a, a, M, K, kPRows)) != DSV3_OK) return rc;
    const bool tma_store = (N % 8) == 0;   // row pitch of the result must be a multiple of 16 bytes for a tensor map
    for (int m = 0; m < kMats; ++m) {
        if ((rc = make_tmap(&ops.b[m], b[m], N, K, kBHalf / 2)) != DSV3_OK) return rc;
        if (tma_store && (rc = make_tmap_out(&ops.c[m], c[m], M, N)) != DSV3_OK) return rc;
    }
    TwParams prm;
    prm.a_s = a_s;
    prm.b_s = b_s[0];
    prm.c = static_cast<__nv_bfloat16*>(c[0]);
    if constexpr (kMats == 2) {
        ops.b_s1 = b_s[1];
        ops.c1 = static_cast<__nv_bfloat16*>(c[1]);
        ops.tiles_q0 = static_cast<int>(tiles_q0);
    }
    prm.status = status_device_ptr();
    if (!prm.status) return DSV3_ERR_CUDA;
    prm.M = M;
    prm.N = N;
    prm.kc = static_cast<int>((K + kChunk - 1) / kChunk);
    prm.nblk = static_cast<int>((N + 127) / 128);
    prm.tiles_pp = static_cast<int>(tiles_pp);
    prm.tiles_q = static_cast<int>(tiles_q);
    // Work order: as many token-tile pairs as keep their activations (raster x 256 x K bytes) within about a
    // quarter of L2 share consecutive weight tiles, so that the weights stream from HBM as few times as possible.
    const int64_t fit = (32ll << 20) / (static_cast<int64_t>(2 * kPRows) * K);
    prm.raster = static_cast<int>(fit < 4 ? 4 : (fit > 32 ? 32 : fit));
    prm.div_raster = make_fast_div(static_cast<uint32_t>(prm.raster));
    prm.div_per_group = make_fast_div(static_cast<uint32_t>(prm.raster) * static_cast<uint32_t>(prm.tiles_q));
    prm.tma_store = tma_store ? 1 : 0;
    const int max_pairs = num_sms() / 2;
    prm.num_tiles = static_cast<int>(tiles_pp * tiles_q);
    prm.tail_tiles = prm.num_tiles % max_pairs;
    prm.tail_w = tw_strip_width(prm.tail_tiles, max_pairs, prm.kc);
    if (prm.tail_w == 0) prm.tail_tiles = 0;
    prm.num_tiles -= prm.tail_tiles;
    for (int m = 0; m < kMats; ++m) {
        ops.s[m] = ops.b[m];
        if (prm.tail_w && (rc = make_tmap(&ops.s[m], b[m], N, K, prm.tail_w / 2)) != DSV3_OK) return rc;
    }

    uintptr_t scales = reinterpret_cast<uintptr_t>(a_s);
    for (int m = 0; m < kMats; ++m) scales |= reinterpret_cast<uintptr_t>(b_s[m]);
    const auto aligned = [&](int n) { return (prm.kc % n) == 0 && (scales % (4 * n)) == 0; };
    auto kern = aligned(4) ? fp8_gemm_tw_kernel<4, kMats> : aligned(2) ? fp8_gemm_tw_kernel<2, kMats>
              : prm.kc >= kShiftedFrom ? fp8_gemm_tw_kernel<kShifted, kMats> : fp8_gemm_tw_kernel<1, kMats>;
    static bool configured[64] = {};
    int dev = 0;
    DSV3_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) {
        set_last_error("fp8_gemm: device ordinal %d is outside the supported range", dev);
        return DSV3_ERR_UNSUPPORTED;
    }
    if (!configured[dev]) {
        DSV3_CUDA_TRY(cudaFuncSetAttribute(fp8_gemm_tw_kernel<4, kMats>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
        DSV3_CUDA_TRY(cudaFuncSetAttribute(fp8_gemm_tw_kernel<2, kMats>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
        DSV3_CUDA_TRY(cudaFuncSetAttribute(fp8_gemm_tw_kernel<kShifted, kMats>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
        DSV3_CUDA_TRY(cudaFuncSetAttribute(fp8_gemm_tw_kernel<1, kMats>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
        configured[dev] = true;
    }
    const int work = prm.num_tiles > 0 && prm.tail_w ? max_pairs : prm.num_tiles + (prm.tail_w ? prm.tail_tiles * (kBN / prm.tail_w) : 0);
    const int pairs = work < max_pairs ? work : max_pairs;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * pairs);
    cfg.blockDim = dim3(kNumThreads);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    DSV3_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, ops, prm));
    return DSV3_OK;
}

}  // namespace

int launch_fp8_gemm_tw(const void* a, const float* a_s, const void* b, const float* b_s, int64_t M, int64_t N, int64_t K, void* c,
                       cudaStream_t stream) {
    return launch<1>(a, a_s, &b, &b_s, M, N, K, &c, stream);
}

int launch_fp8_gemm_tw_two(const void* a, const float* a_s, const void* const (&b)[2], const float* const (&b_s)[2], int64_t M, int64_t N, int64_t K,
                           void* const (&c)[2], cudaStream_t stream) {
    return launch<2>(a, a_s, b, b_s, M, N, K, c, stream);
}

}  // namespace dsv3
