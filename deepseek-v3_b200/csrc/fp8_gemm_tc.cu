// fp8_gemm for sm_100a: TMA-fed, warp-specialised, persistent tcgen05 kernel with
// software promotion of every 128-wide K chunk.
//
// Replaces inference/kernel.py:118-172 (fp8_gemm_kernel) and its launch at :194-195.
//
// Why promotion is done in software: the scales are fp32 (a_s per token per chunk,
// b_s per 128x128 weight block), not ue8m0, so the block-scaled MMA kinds cannot apply
// them.  Each chunk is therefore multiplied into its own TMEM accumulator
// (4 x tcgen05.mma kind::f8f6f4, K = 32 each), read back with tcgen05.ld by the
// promotion warps, and folded into fp32 registers as acc += dot * (a_s * b_s).
//
// The pipeline moves "units" of UC consecutive K chunks, numbered g = 0,1,2,... across all work
// items of a CTA (UC = 2 for token-major tiles, 1 for weight-major tiles):
//   warp 0                   TMA producer: waits empty[g % NS], loads the P and Q tiles of the unit's chunks
//   warps 1,2                MMA issuers, unit g belongs to issuer g % 2: wait tempty[g % NT] and full[g % NS],
//                            issue 4 MMAs per chunk, commit to empty[g % NS] and tfull[g % NT]
//   warps 4..11              promotion: wait tfull[g % NT], read the unit back from TMEM (token-major: both
//                            chunks behind a single tcgen05.wait::ld), release tempty, then do the FMAs; at
//                            the end of a work item write the result (token-major: through shared memory and
//                            a TMA store) or park a split-K partial tile
// Operand roles: P is the 128-row MMA "A" operand, Q the BN-row MMA "B" operand.
//   kSwap = false : P = 128 tokens of a,  Q = 128 or 64 rows of b  (M > 64: "token-major" tiles)
//   kSwap = true  : P = 128 rows of b,    Q = BN tokens of a ("weight-major": M <= 64, where weights stream once; up to 256 tokens on
//                   few weights, in several token tiles, whose smaller parts are exchanged sooner: small_estimate)
// (producer and issuer warps stay converged; one elected lane issues)
// Split-K, up to eight splits: the splits of a tile are the CTAs of one cluster, which exchange rows of the partial tile
// through distributed shared memory and each add a share in split order.  Pinned factors, and more splits: a work item is
// (tile, split), partial tiles go to a workspace and the CTA that takes the last ticket of a tile adds them in split order.
// Both are deterministic; nothing spins.
//
// Hand-off costs set the structure: a dependent mbarrier.try_wait takes ~175 cycles even when the
// phase is already complete and tcgen05.fence::after_thread_sync is of the same order, while a chunk
// is only ~256 cycles of tensor-core work.  So a token-major unit is two chunks, the issue work is split
// over two threads, and every role probes the barrier of its next unit (a non-blocking test_wait whose
// result is consumed one iteration later) where that is safe.
//
// Every wait is bounded: after about a second the waiting thread records what it was
// waiting for in the status word, raises a CTA-wide abort flag and all roles fall
// through to the common teardown (which frees TMEM).
#include <cuda.h>

#include <cstring>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "gemm_plan.cuh"
#include "tc_wait.cuh"

namespace dsv3 {

namespace {

constexpr int kNumThreads = 384;          // warp 0: TMA producer, warps 1-2: MMA issuers, 3 idle, 4..11: promotion
constexpr int kIssuers = 2;
constexpr int kPromoThreads = 256;
constexpr int kFirstPromoWarp = 4;
// Register budget: 384 threads start with 168 each; the control warpgroup gives registers back and
// the two promotion warpgroups take them (64 accumulators + two 64-value read-back buffers).
constexpr int kRegsControl = 40;
constexpr int kRegsPromo = 232;
static_assert(128 * kRegsControl + 256 * kRegsPromo <= 384 * 168, "register pool");

constexpr int kTmemStages = 4;
constexpr int kMaxClusterSplits = 8;      // portable cluster size
constexpr int kMaxTickets = DSV3_WORKSPACE_HEADER_BYTES / 4;

struct TcParams {
    const float* a_s;
    const float* b_s;
    __nv_bfloat16* c;
    float* partials;        // [splits][tiles][bn / 4][128] float4 (padded partial tiles), only when splits > 1
    int* tickets;           // one per tile, zero on entry and on exit
    unsigned int* status;   // device status words
    int64_t M, N;
    int kc;                 // number of K chunks
    int tiles_p, tiles_q;
    int splits;
    int cluster;            // the splits of a tile are the CTAs of one cluster and meet in shared memory (no partials, no tickets)
    FastDiv div_splits, div_per_group, div_raster, div_rows;   // for the work-item decoder
    int raster;             // token-major tiles: P tiles (token tiles) that share consecutive Q tiles in the work order
    int tma_store;          // token-major tiles: results leave through shared memory and a TMA store (needs N % 8 == 0)
    int num_items;          // tiles_p * tiles_q * splits
};

// K chunks of one weight-major work item whose scales fit the shared-memory table: 144 (K <= 18432) for
// 16- and 32-token tiles, 72 for 64-token tiles (the same 18 KB, which leaves room for four 48 KB stages;
// longer K is split)
constexpr int scale_tab_chunks(int bn) { return bn >= 64 ? 72 : 144; }

template <int BN, bool kSwap>
struct Cfg {
    // The pipeline moves "units" of kUC consecutive K chunks: one smem stage, one TMEM stage and one
    // round of hand-offs per unit.  Token-major tiles pair two chunks so that every hand-off (each costs
    // several hundred cycles of latency) covers twice the tensor-core work.
    static constexpr int kUC = (kSwap && BN < 64) ? 1 : 2;
    static constexpr int kChunkBytes = kPRows * kChunk + BN * kChunk;      // P and Q tile of one chunk
    static constexpr int kStageBytes = kUC * kChunkBytes;
    // chunk products resident in TMEM: four 128-column accumulators, or eight of 64 columns
    static constexpr int kAccs = BN == 64 ? 8 : kTmemStages;
    static constexpr int kTmemUnits = kAccs / kUC;                          // unit products resident in TMEM
    // weight-major tiles: a_s * b_s of the item's chunks for the tile's BN tokens, [chunk][token]
    static constexpr int kScaleTabBytes = kSwap ? scale_tab_chunks(BN) * BN * 4 : 0;
    // token-major tiles: the 128 x 128 bf16 result tile is staged here (two 128-byte-swizzled 128 x 64 boxes)
    static constexpr int kStoreBytes = !kSwap && BN == 128 ? kPRows * 128 * 2 : 0;
    // Split-K inside a cluster: partial sums that the other CTAs send here.  16- and 32-token tiles have room of their own
    // for them; the others re-use the operand stages once every CTA of the cluster is through with its own.
    static constexpr bool kOwnExchange = kSwap && BN < 64;
    static constexpr int kExchangeBytes = (kPRows + 10) * BN * 4;    // splits * (ceil(128 / splits) | 1) rows, at most 138
    static constexpr int kStagesRaw =
        (232448 - 2048 - kStoreBytes - kScaleTabBytes - (kOwnExchange ? kExchangeBytes : 0)) / kStageBytes;
    static constexpr int kStagesCap = kStagesRaw > 10 ? 10 : kStagesRaw;
    // weight-major tiles: an even stage count, so that a stage always belongs to the same MMA issuer and
    // the issuer may probe its next full[] barrier (see the issuer loop)
    static constexpr int kStages = kSwap ? (kStagesCap & ~1) : kStagesCap;
    static constexpr int kTmemCols = kAccs * BN;  // 64..512, a power of two
    // tiles + result staging + tables + barriers + control words + slack for the 1024-byte alignment of the tiles
    static constexpr int kSmemBytes =
        kStages * kStageBytes + kStoreBytes + kScaleTabBytes + (kOwnExchange ? kExchangeBytes : 0) + 1024 + 1024;
    static_assert(kOwnExchange || kExchangeBytes <= kStages * kStageBytes, "the exchange fits the operand stages");
    static_assert(kSmemBytes <= 232448, "shared memory per CTA");
    static_assert(kStages >= 3, "at least three smem stages");
    static_assert(kTmemCols >= 32 && kTmemCols <= 512 && (kTmemCols & (kTmemCols - 1)) == 0, "TMEM columns");
    static_assert((BN * kChunk) % 1024 == 0, "Q tile must keep 1024-byte alignment");
    // more than half of an SM's shared memory, so two CTAs can never share an SM (and its TMEM)
    static_assert(kSmemBytes > 116 * 1024, "one CTA per SM");
};

struct Item {
    int p_idx, q_idx, split, tile;
    int c0, c1;     // chunk range
    int row0;       // weight-major tiles: first activation row of the tile
    int row_end;    // weight-major tiles: activation rows at and beyond this index are not part of the problem
};

template <int BN, bool kSwap>
__device__ __forceinline__ Item decode_item(int item, const TcParams& p) {
    Item it;
    it.tile = static_cast<int>(fast_div(static_cast<uint32_t>(item), p.div_splits));
    it.split = item - it.tile * p.splits;
    // work order: `raster` P tiles share consecutive Q tiles so that a wave re-uses both operands in L2
    const int kGroup = p.raster;
    const int per_group = kGroup * p.tiles_q;
    const int grp = static_cast<int>(fast_div(static_cast<uint32_t>(it.tile), p.div_per_group));
    const int first_p = grp * kGroup;
    const int gsz = min(kGroup, p.tiles_p - first_p);
    const int r = it.tile - grp * per_group;
    it.q_idx = (gsz == kGroup) ? static_cast<int>(fast_div(static_cast<uint32_t>(r), p.div_raster)) : r / gsz;   // the last group may be shorter
    it.p_idx = first_p + (r - it.q_idx * gsz);
    // kc * split < 2^31 (kc < 2^24, at most 64 splits)
    it.c0 = static_cast<int>(fast_div(static_cast<uint32_t>(p.kc * it.split), p.div_splits));
    it.c1 = static_cast<int>(fast_div(static_cast<uint32_t>(p.kc * (it.split + 1)), p.div_splits));
    it.row0 = it.q_idx * BN;
    it.row_end = static_cast<int>(p.M);
    return it;
}

template <int N>
__device__ __forceinline__ void tmem_load_cols(uint32_t taddr, uint32_t* v) {
    if constexpr (N == 8) {
        tc_ld_x8(taddr, v);
    } else if constexpr (N == 16) {
        tc_ld_x16(taddr, v);
    } else if constexpr (N == 32) {
        tc_ld_x32(taddr, v);
    } else {
        static_assert(N == 64, "columns per thread");
        tc_ld_x32(taddr, v);
        tc_ld_x32(taddr + 32, v + 32);
    }
}

// Barrier among the threads that write results (promotion group 0, or all promotion warps when
// there is a single group).
template <int kThreads>
__device__ __forceinline__ void promo_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory"); }

template <int BN, bool kSwap>
__global__ void __launch_bounds__(kNumThreads, 1)
fp8_gemm_tc_kernel(const __grid_constant__ CUtensorMap tmap_p, const __grid_constant__ CUtensorMap tmap_q,
                   const __grid_constant__ CUtensorMap tmap_c, const TcParams p) {
    using C = Cfg<BN, kSwap>;
    constexpr int NS = C::kStages;
    constexpr int UC = C::kUC;           // K chunks per pipeline unit
    constexpr int NT = C::kTmemUnits;    // TMEM stages, in units
    constexpr int CPT = BN / 2;       // accumulator columns per promotion thread (a thread owns half a row)
    constexpr int kWriters = kPromoThreads;
    static_assert(kSwap || BN == 128 || BN == 64, "token-major tiles are 128 x 128 or 128 x 64: one b_s value per tile and chunk");

    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t tiles = (raw + 1023u) & ~1023u;
    uint8_t* gen_tiles = smem_raw + (tiles - raw);
    uint8_t* store_buf = gen_tiles + NS * C::kStageBytes;                       // 1024-byte aligned (swizzle atom)
    uint8_t* after_store = store_buf + C::kStoreBytes;
    float* sc_tab = reinterpret_cast<float*>(after_store);   // [chunk][token]
    float* exchange = reinterpret_cast<float*>(C::kOwnExchange ? after_store + C::kScaleTabBytes : gen_tiles);
    uint64_t* bars = reinterpret_cast<uint64_t*>(after_store + C::kScaleTabBytes + (C::kOwnExchange ? C::kExchangeBytes : 0));
    Control* ctl = reinterpret_cast<Control*>(bars + 2 * NS + 2 * NT + 2);
    const uint32_t bar0 = smem_u32(bars);
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (NS + s); };
    auto tfull_bar = [&](int s) { return bar0 + 8u * (2 * NS + s); };
    auto tempty_bar = [&](int s) { return bar0 + 8u * (2 * NS + NT + s); };
    const uint32_t tab_ready_bar = bar0 + 8u * (2 * NS + 2 * NT);       // scale table of the item is filled
    const uint32_t tab_free_bar = bar0 + 8u * (2 * NS + 2 * NT + 1);    // scale table may be overwritten

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);   // uniform, and known to be
    const int lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int s = 0; s < NT; ++s) {
            mbar_init(tfull_bar(s), 1);
            mbar_init(tempty_bar(s), kPromoThreads / 32);   // every promotion warp reads every stage
        }
        mbar_init(tab_ready_bar, kPromoThreads);
        mbar_init(tab_free_bar, kPromoThreads);
        ctl->abort_flag = 0;
        ctl->ticket[0] = 0;
        ctl->ticket[1] = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmap_p);
        tma_prefetch_desc(&tmap_q);
        if (!kSwap && p.tma_store) tma_prefetch_desc(&tmap_c);
    }
    if (warp == 1) tc_alloc(smem_u32(&ctl->tmem_base), C::kTmemCols);
    // Programmatic dependent launch: nothing above touches global memory, so it may overlap the tail of
    // the kernel before this one in the stream.  While waiting for that kernel, the producer thread pulls
    // the first weight boxes of this CTA's first work item into L2 (L2 is the point of coherence: should
    // the predecessor still be writing those weights, the later TMA loads see its data all the same).
    if (threadIdx.x == 0 && static_cast<int>(blockIdx.x) < p.num_items) {
        const Item it = decode_item<BN, kSwap>(blockIdx.x, p);
        const void* wmap = kSwap ? static_cast<const void*>(&tmap_p) : static_cast<const void*>(&tmap_q);
        const int wrow = kSwap ? it.p_idx * kPRows : it.q_idx * BN;
        const int n_pre = min(it.c1 - it.c0, NS * UC);
        for (int j = 0; j < n_pre; ++j) tma_prefetch_l2_2d(wmap, (it.c0 + j) * kChunk, wrow);
    }
    griddep_launch_dependents();
    griddep_wait();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = ctl->tmem_base;
    if (C::kOwnExchange && p.cluster) cluster_arrive();             // waited for in front of the exchange

    bool exchanged = false;
    if constexpr (!kSwap) {
        if (warp < kFirstPromoWarp) {
            asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsControl));
        } else {
            asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsPromo));
        }
    }

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        // The whole warp walks the loop (waits included) and one elected lane issues: control flow, addresses and
        // descriptors then stay warp-uniform, which is what makes TMA and tcgen05 instructions cheap to issue.
        {
            uint32_t g = 0;
            uint32_t probe = 0;   // result of try_wait on empty[] for chunk g, issued one chunk earlier
            bool ok = true;
            for (int item = blockIdx.x; ok && item < p.num_items; item += gridDim.x) {
                const Item it = decode_item<BN, kSwap>(item, p);
                const int p_row = it.p_idx * kPRows;
                const int q_row = kSwap ? it.row0 : it.q_idx * BN;
                const int n_units = (it.c1 - it.c0 + UC - 1) / UC;
                for (int u = 0; u < n_units; ++u, ++g) {
                    const int s = g % NS;
                    ok = __all_sync(0xffffffffu, wait_probed(probe, empty_bar(s), ((g / NS) & 1u) ^ 1u, ctl, p.status, 1, g));
                    if (!ok) break;
                    probe = mbar_test_wait(empty_bar((g + 1) % NS), (((g + 1) / NS) & 1u) ^ 1u) ? 1u : 0u;
                    const int k0 = it.c0 + u * UC;
                    const int nch = min(UC, it.c1 - k0);
                    if (elect_one()) {
                        mbar_arrive_expect_tx(full_bar(s), nch * C::kChunkBytes);
                        for (int j = 0; j < nch; ++j) {
                            const uint32_t dst = tiles + s * C::kStageBytes + j * C::kChunkBytes;
                            tma_load_2d(dst, &tmap_p, (k0 + j) * kChunk, p_row, full_bar(s));
                            tma_load_2d(dst + kPRows * kChunk, &tmap_q, (k0 + j) * kChunk, q_row, full_bar(s));
                        }
                    }
                    __syncwarp();
                }
            }
            // Nothing waits for the commits onto the empty[] barriers of the last units; wait for them here so
            // that none is in flight when the CTA leaves (it would land in whatever CTA gets this shared memory next).
            for (uint32_t d = (g > static_cast<uint32_t>(NS) ? g - NS : 0u); ok && d < g; ++d)
                ok = __all_sync(0xffffffffu, bounded_wait(empty_bar(d % NS), (d / NS) & 1u, ctl, p.status, 1, d));
        }
    } else if (warp <= kIssuers) {
        // ------------------------------------------------------------ MMA issuers (chunk g -> issuer g % kIssuers)
        // (converged warp, elected lane: see the producer)
        {
            constexpr uint32_t idesc = umma_idesc_e4m3_f32(kPRows, BN);
            const uint32_t me = static_cast<uint32_t>(warp - 1);
            uint32_t g = 0;
            uint32_t probe_t = 0, probe_f = 0;   // probes of tempty[] / full[] for this issuer's next unit
            bool ok = true;
            for (int item = blockIdx.x; ok && item < p.num_items; item += gridDim.x) {
                const Item it = decode_item<BN, kSwap>(item, p);
                const int n_units = (it.c1 - it.c0 + UC - 1) / UC;
                for (int u = 0; u < n_units; ++u, ++g) {
                    if (g % kIssuers != me) continue;
                    const int s = g % NS, ts = g % NT;
                    constexpr bool kProbeFull = (NS % kIssuers) == 0;
                    ok = __all_sync(0xffffffffu, wait_probed(probe_t, tempty_bar(ts), ((g / NT) & 1u) ^ 1u, ctl, p.status, 3, g) &&
                                                 wait_probed(kProbeFull ? probe_f : 0u, full_bar(s), (g / NS) & 1u, ctl, p.status, 2, g));
                    if (!ok) break;
                    {   // Probe the TMEM stage of this issuer's next unit now; the answer is read one iteration
                        // later.  A parity probe is only meaningful if the barrier's previous phase is known to be
                        // complete: true for tempty (NT is even, so a stage always belongs to the same issuer, which
                        // waited for that phase itself); for full[] only when NS is even as well (otherwise the previous
                        // phase of that stage belongs to the other issuer and the barrier is always waited for).
                        static_assert(NT % kIssuers == 0, "a TMEM stage must always be used by the same issuer");
                        const uint32_t gn = g + kIssuers;
                        probe_t = mbar_test_wait(tempty_bar(gn % NT), ((gn / NT) & 1u) ^ 1u) ? 1u : 0u;
                        if constexpr (kProbeFull) probe_f = mbar_test_wait(full_bar(gn % NS), (gn / NS) & 1u) ? 1u : 0u;
                    }
                    tc_fence_after();
                    const int nch = min(UC, it.c1 - it.c0 - u * UC);
                    if (elect_one()) {
                        for (int j = 0; j < nch; ++j) {
                            const uint32_t sp = tiles + s * C::kStageBytes + j * C::kChunkBytes;
                            const uint64_t dp = umma_desc_k_major_sw128(sp);
                            const uint64_t dq = umma_desc_k_major_sw128(sp + kPRows * kChunk);
                            const uint32_t d_tmem = tmem_base + (ts * UC + j) * BN;   // one TMEM region per chunk
#pragma unroll
                            for (int k = 0; k < kChunk / 32; ++k) {
                                // 32 bytes further along K inside the 128-byte swizzle atom: +2 in address units of 16 B
                                tc_mma_f8(d_tmem, dp + 2u * k, dq + 2u * k, idesc, k > 0 ? 1u : 0u);
                            }
                        }
                        tc_commit(empty_bar(s));   // smem stage reusable once these MMAs have read it
                        tc_commit(tfull_bar(ts));  // the unit's chunk products are complete in TMEM
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp >= kFirstPromoWarp) {
        // ------------------------------------------------------------ promotion + epilogue
        // All eight warps work on every unit: warps 4..7 own the left half of the tile's columns, warps 8..11
        // the right half; within a half, a thread owns one accumulator row (TMEM lane) and CPT columns.
        const int col0 = ((warp - kFirstPromoWarp) >> 2) * CPT;
        const int quarter = warp & 3;                       // TMEM lane quarter this warp may access
        const int row = quarter * 32 + lane;                // accumulator row (TMEM lane)
        const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + col0;
        const int64_t M = p.M, N = p.N;
        const int kc = p.kc;
        uint32_t g = 0;          // unit counter at the start of the current item
        uint32_t item_no = 0;    // non-empty items done by this CTA (phase of the scale-table barriers, ticket slot)
        bool ok = true;

        // A chunk is read back in SPC steps of HC columns so that one step's TMEM load is in flight
        // while the previous step's FMAs issue.
        constexpr int HC = (CPT >= 32) ? 32 : CPT;
        constexpr int SPC = CPT / HC;
        uint32_t probe = 0;   // result of test_wait on tfull[] for the next unit
        // token-major tiles: two read-back buffers of one chunk (64 columns) each
        constexpr bool kBatched = !kSwap;
        uint32_t va64[kBatched ? CPT : 1], vb64[kBatched ? CPT : 1];
        auto load_chunk = [](uint32_t taddr, uint32_t* v) {
            if constexpr (CPT == 64) tc_ld_x64(taddr, v);
            else if constexpr (CPT == 32) tc_ld_x32(taddr, v);
        };
        // Issues (does not wait for) the load of step `st` of chunk `j` of unit `gu`; the first step of a
        // unit first waits for the unit's products to be complete in TMEM.
        auto issue_load = [&](uint32_t gu, int j, int st, uint32_t* v) -> bool {
            const int ts = gu % NT;
            if (j == 0 && st == 0) {
                const bool mine = wait_probed(probe, tfull_bar(ts), (gu / NT) & 1u, ctl, p.status, 4, gu);
                if (!__all_sync(0xffffffffu, mine)) return false;
                probe = mbar_test_wait(tfull_bar((gu + 1) % NT), ((gu + 1) / NT) & 1u) ? 1u : 0u;
                tc_fence_after();
            }
            tmem_load_cols<HC>(t_lane + (ts * UC + j) * BN + st * HC, v);
            return true;
        };
        // Completes the outstanding load; `last` = it was the last load of the unit, whose TMEM stage
        // then goes back to the MMA issuers.
        auto finish_load = [&](uint32_t gu, bool last) {
            tc_wait_ld();
            if (last) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tempty_bar(gu % NT));
            }
        };

        for (int item = blockIdx.x; item < p.num_items; item += gridDim.x) {
            const Item it = decode_item<BN, kSwap>(item, p);
            const uint32_t item_cur = item_no++;
            float2 acc[CPT / 2];
#pragma unroll
            for (int j = 0; j < CPT / 2; ++j) acc[j] = make_float2(0.0f, 0.0f);

            // token / weight-row coordinates of this thread
            const int64_t p_row = static_cast<int64_t>(it.p_idx) * kPRows + row;
            const int64_t q_base = (kSwap ? static_cast<int64_t>(it.row0) : static_cast<int64_t>(it.q_idx) * BN) + col0;
            const int64_t m_end = kSwap ? static_cast<int64_t>(it.row_end) : M;   // weight-major: token rows of this item end here
            const float* as_ptr;  // normal: this row's scales ; swap: scale matrix, indexed per token below
            const float* bs_ptr;
            if constexpr (!kSwap) {
                as_ptr = p.a_s + min(p_row, M - 1) * kc;
                bs_ptr = p.b_s + static_cast<int64_t>(it.q_idx) * BN / 128 * kc;
            } else {
                as_ptr = p.a_s;
                bs_ptr = p.b_s + static_cast<int64_t>(it.p_idx) * kc;        // 128 weight rows = one scale row
            }
            const int n_ch = it.c1 - it.c0;
            // Weight-major tiles: every thread needs a_s * b_s of all its tokens for every chunk; the
            // promotion warps put them into shared memory once per item ([chunk][token]) so that the
            // chunk loop reads them with a few broadcast vector loads.  (The host plan splits K so that an
            // item never has more chunks than the table holds.)
            if constexpr (kSwap) {
                if (ok) {
                    const bool mine = bounded_wait(tab_free_bar, (item_cur & 1u) ^ 1u, ctl, p.status, 7, item_cur);
                    ok = __all_sync(0xffffffffu, mine);
                }
                if (ok) {
                    const int tid = threadIdx.x - kFirstPromoWarp * 32;
                    for (int idx = tid; idx < n_ch * BN; idx += kPromoThreads) {
                        const int chl = idx / BN, col = idx - chl * BN;
                        const int64_t m = max(min(static_cast<int64_t>(it.row0) + col, m_end - 1), static_cast<int64_t>(0));
                        sc_tab[idx] = __ldg(as_ptr + m * kc + it.c0 + chl) * __ldg(bs_ptr + it.c0 + chl);
                    }
                    mbar_arrive(tab_ready_bar);
                    const bool mine = bounded_wait(tab_ready_bar, item_cur & 1u, ctl, p.status, 8, item_cur);
                    ok = __all_sync(0xffffffffu, mine);
                }
            }
            const int n_units = (n_ch + UC - 1) / UC;
            const int n_mine = n_units;
            auto unit_g = [&](int mu) -> uint32_t { return g + mu; };                        // pipeline counter
            auto unit_k = [&](int mu) -> int { return it.c0 + UC * mu; };                    // first K chunk of the unit
            auto unit_n = [&](int mu) -> int { return min(UC, it.c1 - unit_k(mu)); };        // chunks in the unit
            // acc[off ..] += v * (a_s * b_s) for K chunk ch; v holds HC columns starting at column 2*off
            auto fold = [&](int ch, const uint32_t* v, float sc, auto off_c) {
                constexpr int off = decltype(off_c)::value;
                if constexpr (!kSwap) {
                    const float2 sc2 = make_float2(sc, sc);
#pragma unroll
                    for (int j = 0; j < HC / 2; ++j)
                        acc[off + j] = __ffma2_rn(make_float2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])),
                                                  sc2, acc[off + j]);
                } else {
                    const float2* t2 = reinterpret_cast<const float2*>(sc_tab + (ch - it.c0) * BN + col0) + off;
#pragma unroll
                    for (int j = 0; j < HC / 2; ++j)
                        acc[off + j] = __ffma2_rn(make_float2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])),
                                                  t2[j], acc[off + j]);
                }
            };

            // Software pipeline over the load steps, two register buffers: while the FMAs of one step issue,
            // the TMEM load of the next step is in flight.
            uint32_t va[kBatched ? 1 : HC], vb[kBatched ? 1 : HC];
            if constexpr (kBatched) {
                if (ok && n_mine > 0) {   // first unit of the item: wait and start its first load here
                    const uint32_t gu = unit_g(0);
                    const bool mine = wait_probed(probe, tfull_bar(gu % NT), (gu / NT) & 1u, ctl, p.status, 4, gu);
                    ok = __all_sync(0xffffffffu, mine);
                    if (ok) {
                        tc_fence_after();
                        load_chunk(t_lane + ((gu % NT) * UC) * BN, va64);
                    }
                }
            } else {
                if (ok && n_mine > 0) ok = issue_load(unit_g(0), 0, 0, va);
            }
            if constexpr (!kSwap) {
                static_assert(UC == 2, "token-major tiles pair two chunks per unit");
                // ---- token-major tiles: a thread reads its 64 columns of both
                // chunks of the unit in one batch (tcgen05.wait::ld has no per-load granularity, so one wait
                // per unit exposes the TMEM latency once), returns the TMEM stage at once and only then does
                // the FMAs; the other promotion warp of the scheduler overlaps with them.  Row scales (global
                // memory) are fetched one unit ahead.
                // raw scales one unit ahead, multiplied when the unit begins (see fp8_gemm_tm.cu)
                float ra0, ra1, rb0, rb1;
                auto load_scales = [&](int k) {        // clamped so that the look-ahead never leaves the item
                    const int c0 = min(k, it.c1 - 1), c1 = min(k + 1, it.c1 - 1);
                    ra0 = __ldg(as_ptr + c0);
                    ra1 = __ldg(as_ptr + c1);
                    rb0 = __ldg(bs_ptr + c0);
                    rb1 = __ldg(bs_ptr + c1);
                };
                load_scales(unit_k(0));
                for (int mu = 0; ok && mu < n_mine; ++mu) {
                    const uint32_t gu = unit_g(mu);
                    const int ts = gu % NT;
                    const int nch = unit_n(mu);
                    if (mu > 0) {
                        const bool mine = wait_probed(probe, tfull_bar(ts), (gu / NT) & 1u, ctl, p.status, 4, gu);
                        ok = __all_sync(0xffffffffu, mine);
                        if (!ok) break;
                        tc_fence_after();
                    }
                    const uint32_t taddr = t_lane + (ts * UC) * BN;
                    if (mu > 0) load_chunk(taddr, va64);
                    if (nch > 1) load_chunk(taddr + BN, vb64);
                    const float sa0 = ra0 * rb0, sa1 = ra1 * rb1;
                    load_scales(unit_k(mu + 1));
                    tc_wait_ld();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(tempty_bar(ts));
                    // probe the next unit now: its answer is needed only after the FMAs below, by which time
                    // the probe has long returned (and the unit's MMAs, issued a unit ago, are usually complete)
                    probe = mbar_test_wait(tfull_bar((gu + 1) % NT), ((gu + 1) / NT) & 1u) ? 1u : 0u;
                    {
                        const float2 sc2 = make_float2(sa0, sa0);
#pragma unroll
                        for (int j = 0; j < CPT / 2; ++j)
                            acc[j] = __ffma2_rn(make_float2(__uint_as_float(va64[2 * j]), __uint_as_float(va64[2 * j + 1])),
                                                sc2, acc[j]);
                    }
                    if (nch > 1) {
                        const float2 sc2 = make_float2(sa1, sa1);
#pragma unroll
                        for (int j = 0; j < CPT / 2; ++j)
                            acc[j] = __ffma2_rn(make_float2(__uint_as_float(vb64[2 * j]), __uint_as_float(vb64[2 * j + 1])),
                                                sc2, acc[j]);
                    }
                }
            } else {
                // ---- weight-major tiles: a unit is one chunk (16- and 32-token tiles) or two (64-token tiles);
                // a chunk is read back in SPC steps, one trip covers max(2, SPC) steps
                constexpr int U = SPC > 2 ? SPC : 2;
                const int n_steps = n_ch * SPC;
                auto step = [&](int t, auto u_c, uint32_t* cur, uint32_t* nxt) {
                    constexpr int u = decltype(u_c)::value;
                    constexpr int st = u % SPC;
                    const int T = t + u;
                    if (!ok || T >= n_steps) return;
                    const int c = T / SPC;                              // chunk of the item
                    const bool last_of_unit = (st == SPC - 1) && ((c % UC) == UC - 1 || c == n_ch - 1);
                    finish_load(unit_g(c / UC), last_of_unit);
                    if (T + 1 < n_steps) {
                        const int cn = (T + 1) / SPC;
                        ok = issue_load(unit_g(cn / UC), cn % UC, (u + 1) % SPC, nxt);
                    }
                    fold(it.c0 + c, cur, 0.0f, std::integral_constant<int, st * (HC / 2)>{});
                };
                for (int t = 0; ok && t < n_steps; t += U) {
                    step(t, std::integral_constant<int, 0>{}, va, vb);
                    step(t, std::integral_constant<int, 1>{}, vb, va);
                    if constexpr (U == 4) {
                        step(t, std::integral_constant<int, 2>{}, va, vb);
                        step(t, std::integral_constant<int, 3>{}, vb, va);
                    }
                }
            }
            g += n_units;
            // A warp whose wait gave up goes on through the items without working on them, to take part in the barriers
            // where other warps may be waiting for it (barrier_all); the cluster's barriers come behind the loop.
            if (!ok && (p.cluster || (p.splits == 1 && (kSwap || !p.tma_store)))) break;
            if constexpr (kSwap) {
                if (ok) mbar_arrive(tab_free_bar);   // this thread is done reading the scale table
            }

            float* accf = reinterpret_cast<float*>(acc);

            // ---------------------------------------------------- write-out
            // normal: thread = token row, CPT consecutive output columns
            // swap  : thread = output column (weight row), CPT tokens
            bool write_out = true;
            if (p.cluster) {
                // Split-K inside a cluster (one item per CTA).  CTA r of the cluster adds up and writes rows
                // [r R, (r+1) R) of the tile, R = ceil(128 / splits): every CTA sends each peer its rows of the partial
                // tile (st.shared::cluster), a cluster barrier later everybody adds what arrived, in split order.
                // Against the ticket form below (partial tiles through L2, an atomic, the last arrival reads
                // everything back) this takes about 1.5 us off a launch.
                // A peer is reached in 512-byte runs: a store per row, 16 bytes at a time, made the same exchange 1.1 us
                // slower for 128-token tiles and 0.6 us for 64 (7168 -> 576 at M = 256 10.5 -> 9.2, at M = 64 7.4 -> 6.7).
                const int S = p.splits, R = (kPRows + S - 1) / S;
                if constexpr (!C::kOwnExchange) cluster_arrive();   // through with the operand stages
                cluster_wait();                                     // every CTA runs, and with shared stages is through with them
                const int dest = static_cast<int>(fast_div(static_cast<uint32_t>(row), p.div_rows)), r_local = row - dest * R;
                const uint32_t remote = mapa_shared(smem_u32(exchange), static_cast<uint32_t>(dest));
                const int ntok = static_cast<int>(min(static_cast<int64_t>(BN), m_end - (q_base - col0)));   // weight-major tiles
                // [split][four columns][R | 1 rows] float4: the lanes of a store are consecutive rows, 512 contiguous bytes on
                // their way to the peer
                const int Rp = R | 1;
                const uint32_t at = remote + 16u * ((it.split * (BN / 4) + col0 / 4) * Rp + r_local);
#pragma unroll
                for (int j = 0; j < CPT / 4; ++j)
                    if (!kSwap || col0 + 4 * j < ntok)
                        asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(at + 16u * j * Rp), "f"(accf[4 * j]), "f"(accf[4 * j + 1]),
                                     "f"(accf[4 * j + 2]), "f"(accf[4 * j + 3]) : "memory");
                cluster_arrive();
                cluster_wait();
                const int me = static_cast<int>(cluster_ctarank()), rows_here = min(R, kPRows - me * R);
                const int tid = threadIdx.x - kFirstPromoWarp * 32;
                if constexpr (kSwap) {
                    // a thread adds four tokens of one row; neighbouring threads take neighbouring rows (output columns)
                    const int64_t n0 = static_cast<int64_t>(it.p_idx) * kPRows + me * R;
                    for (int e = tid; e < (ntok + 3) / 4 * R; e += kPromoThreads) {
                        const int t4 = static_cast<int>(fast_div(static_cast<uint32_t>(e), p.div_rows)), i = e - t4 * R;
                        if (i >= rows_here || n0 + i >= N) continue;
                        const float4* src = reinterpret_cast<const float4*>(exchange) + t4 * Rp + i;
                        float4 sum = *src;
                        for (int sp = 1; sp < S; ++sp) {
                            const float4 a = src[sp * (BN / 4) * Rp];
                            sum.x += a.x; sum.y += a.y; sum.z += a.z; sum.w += a.w;
                        }
                        __nv_bfloat16* dst = p.c + (static_cast<int64_t>(it.row0) + 4 * t4) * N + n0 + i;
                        const float v4[4] = {sum.x, sum.y, sum.z, sum.w};
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            if (4 * t4 + q < ntok) dst[q * N] = __float2bfloat16_rn(v4[q]);
                    }
                } else {
                    const bool vec_ok = (N % 8) == 0;
                    for (int e = tid; e < rows_here * (BN / 8); e += kPromoThreads) {      // eight columns each
                        const int i = e / (BN / 8), k8 = e % (BN / 8), r_tile = me * R + i;
                        const int64_t m = static_cast<int64_t>(it.p_idx) * kPRows + r_tile, n = static_cast<int64_t>(it.q_idx) * BN + 8 * k8;
                        if (m >= M || n >= N) continue;
                        float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
                        for (int sp = 0; sp < S; ++sp) {
                            const float4* src = reinterpret_cast<const float4*>(exchange) + (sp * (BN / 4) + 2 * k8) * Rp + i;
                            const float4 a = src[0], b = src[Rp];
                            lo.x += a.x; lo.y += a.y; lo.z += a.z; lo.w += a.w;
                            hi.x += b.x; hi.y += b.y; hi.z += b.z; hi.w += b.w;
                        }
                        __nv_bfloat16* dst = p.c + m * N + n;
                        if (vec_ok && n + 8 <= N) {
                            *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16x2(lo.x, lo.y), pack_bf16x2(lo.z, lo.w), pack_bf16x2(hi.x, hi.y), pack_bf16x2(hi.z, hi.w));
                        } else {
                            const float v8[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
                            for (int q = 0; q < 8; ++q)
                                if (n + q < N) dst[q] = __float2bfloat16_rn(v8[q]);
                        }
                    }
                }
                write_out = false;
                exchanged = true;
            } else if (p.splits > 1) {
                // Split-K: park the partial sums, take a ticket; the last arrival of the tile sums the
                // partial tiles in split order (deterministic) and writes the result.  Partial tiles use a
                // private layout chosen for coalescing, [split][tile][group of 4 columns][128 rows] float4:
                // a warp (32 consecutive rows, one column group) moves 512 contiguous bytes, and rows and
                // columns beyond M or N are stored like the rest, so nothing here is predicated and the
                // compiler is free to keep a whole batch of loads in flight.
                constexpr int kTileVec = BN * kPRows / 4;
                const int64_t split_stride = static_cast<int64_t>(p.tiles_p) * p.tiles_q * kTileVec;
                float4* tile_part = reinterpret_cast<float4*>(p.partials) + static_cast<int64_t>(it.tile) * kTileVec +
                                    (col0 / 4) * kPRows + row;
                if (ok) {
                    float4* dst = tile_part + it.split * split_stride;
#pragma unroll
                    for (int j = 0; j < CPT / 4; ++j)
                        __stcg(dst + j * kPRows, make_float4(accf[4 * j], accf[4 * j + 1], accf[4 * j + 2], accf[4 * j + 3]));
                }
                // Release: the barrier orders every writer's stores before the ticket thread's fence, which
                // is cumulative.  The ticket slot alternates between items, so the next item's ticket cannot
                // overwrite this one before every thread has read it (a barrier of the next item lies between).
                const int slot = static_cast<int>(item_cur & 1u);
                ok = barrier_all<kWriters>(1, ok);
                if (!ok) break;                  // all eight warps
                if (threadIdx.x == kFirstPromoWarp * 32) {
                    // one acquire-release atomic: releases the partial tiles (cumulative over the barrier above) and
                    // acquires the other splits' tiles for the reads below
                    int t;
                    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(t) : "l"(p.tickets + it.tile) : "memory");
                    if (t == p.splits - 1) p.tickets[it.tile] = 0;  // last arrival: leave the ticket clean
                    ctl->ticket[slot] = t;
                }
                promo_barrier<kWriters>();
                write_out = (ctl->ticket[slot] == p.splits - 1);
                if (write_out) {
#pragma unroll
                    for (int j = 0; j < CPT; ++j) accf[j] = 0.0f;
                    constexpr int kBatch = (CPT >= 64) ? 1 : 64 / CPT;   // splits whose loads are in flight together (64 registers)
                    for (int sp0 = 0; sp0 < p.splits; sp0 += kBatch) {
                        float4 t4[kBatch][CPT / 4];
#pragma unroll
                        for (int bi = 0; bi < kBatch; ++bi) {
                            const float4* src = tile_part + min(sp0 + bi, p.splits - 1) * split_stride;
#pragma unroll
                            for (int j = 0; j < CPT / 4; ++j) t4[bi][j] = __ldcg(src + j * kPRows);
                        }
#pragma unroll
                        for (int bi = 0; bi < kBatch; ++bi) {
                            if (sp0 + bi < p.splits) {
#pragma unroll
                                for (int j = 0; j < CPT / 4; ++j) {
                                    accf[4 * j] += t4[bi][j].x;
                                    accf[4 * j + 1] += t4[bi][j].y;
                                    accf[4 * j + 2] += t4[bi][j].z;
                                    accf[4 * j + 3] += t4[bi][j].w;
                                }
                            }
                        }
                    }
                }
            }
            if (write_out) {
                if constexpr (!kSwap) {
                    if (BN == 128 && p.tma_store) {
                        // The four warps of a column half stage their 128 x 64 bf16 box in shared memory (128-byte
                        // swizzle: 16-byte slot c of row r sits at slot c ^ (r & 7), which also keeps the
                        // vector stores free of bank conflicts) and one thread hands it to the TMA, which clips
                        // rows beyond M and columns beyond N.  The store of the previous tile is only known to
                        // have read the buffer once its issuer has waited for it, hence the first barrier.
                        static_assert(BN != 128 || CPT == 64, "one 128-byte box row per thread");
                        const int half = (warp - kFirstPromoWarp) >> 2;
                        uint8_t* sbuf = store_buf + half * (kPRows * 128);
                        const bool issuer = ((threadIdx.x & 127) == 0);
                        if (issuer) bulk_wait_group_read0();
                        ok = barrier_all<128>(2 + half, ok);
                        if (!ok) break;          // this half's four warps (unsplit: no barrier counts all eight)
#pragma unroll
                        for (int cidx = 0; cidx < CPT / 8; ++cidx) {
                            const int j = cidx * 8;
                            const uint4 o = make_uint4(pack_bf16x2(accf[j], accf[j + 1]), pack_bf16x2(accf[j + 2], accf[j + 3]),
                                                       pack_bf16x2(accf[j + 4], accf[j + 5]), pack_bf16x2(accf[j + 6], accf[j + 7]));
                            *reinterpret_cast<uint4*>(sbuf + row * 128 + ((cidx ^ (row & 7)) << 4)) = o;
                        }
                        fence_proxy_async_shared();
                        asm volatile("bar.sync %0, 128;" ::"r"(2 + half) : "memory");
                        if (issuer) {
                            tma_store_2d(&tmap_c, smem_u32(sbuf), it.q_idx * BN + half * 64, it.p_idx * kPRows);
                            bulk_commit_group();
                        }
                    } else if (p_row < M) {
                        __nv_bfloat16* crow = p.c + p_row * N;
                        const bool vec_ok = (N % 8) == 0;
#pragma unroll
                        for (int j = 0; j < CPT; j += 8) {
                            const int64_t n = q_base + j;
                            if (vec_ok && n + 8 <= N) {
                                uint4 o = make_uint4(pack_bf16x2(accf[j], accf[j + 1]), pack_bf16x2(accf[j + 2], accf[j + 3]),
                                                     pack_bf16x2(accf[j + 4], accf[j + 5]), pack_bf16x2(accf[j + 6], accf[j + 7]));
                                *reinterpret_cast<uint4*>(crow + n) = o;
                            } else {
#pragma unroll
                                for (int e = 0; e < 8; ++e)
                                    if (n + e < N) crow[n + e] = __float2bfloat16_rn(accf[j + e]);
                            }
                        }
                    }
                } else {
                    if (p_row < N) {
#pragma unroll
                        for (int j = 0; j < CPT; ++j) {
                            const int64_t m = q_base + j;
                            if (m < m_end) p.c[m * N + p_row] = __float2bfloat16_rn(accf[j]);
                        }
                    }
                }
            }
        }
    }

    // The cluster barriers of the split-K exchange count every thread: the control warps pass through them here, and so
    // does a promotion warp whose wait gave up.
    if (p.cluster && (warp < kFirstPromoWarp || !exchanged)) {
        __syncwarp();
        if constexpr (!C::kOwnExchange) cluster_arrive();
        cluster_wait();
        cluster_arrive();
        cluster_wait();
    }

    // ---------------------------------------------------------------- teardown
    if (!kSwap && warp >= kFirstPromoWarp && (threadIdx.x & 127) == 0) bulk_wait_group0();   // result tiles have left shared memory
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
    if (warp == 1) {
        tc_fence_after();
        tc_dealloc(tmem_base, C::kTmemCols);
    }
}

// -------------------------------------------------------------------- host side

}  // namespace

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(ptr);
    });
    return fn;
}

// [rows, K] bytes, row-major; box = 128 bytes x box_rows, 128-byte swizzle, zero fill outside.
int make_tmap(CUtensorMap* map, const void* base, int64_t rows, int64_t K, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) {
        set_last_error("cuTensorMapEncodeTiled is not available from the driver");
        return DSV3_ERR_CUDA;
    }
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(K)};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(kChunk), static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_last_error("cuTensorMapEncodeTiled failed with CUresult %d (rows=%lld K=%lld box_rows=%d)", static_cast<int>(r),
                       static_cast<long long>(rows), static_cast<long long>(K), box_rows);
        return DSV3_ERR_CUDA;
    }
    return DSV3_OK;
}

// Result matrix [M, N] bf16, row-major; box = 64 columns (128 bytes) x box_rows rows, 128-byte swizzle.
int make_tmap_out(CUtensorMap* map, void* base, int64_t M, int64_t N, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) {
        set_last_error("cuTensorMapEncodeTiled is not available from the driver");
        return DSV3_ERR_CUDA;
    }
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(N), static_cast<cuuint64_t>(M)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(N) * 2};
    const cuuint32_t box[2] = {64, static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, base, dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_last_error("cuTensorMapEncodeTiled (result matrix) failed with CUresult %d (M=%lld N=%lld)", static_cast<int>(r),
                       static_cast<long long>(M), static_cast<long long>(N));
        return DSV3_ERR_CUDA;
    }
    return DSV3_OK;
}

namespace {

template <int BN, bool kSwap>
int launch_variant(const CUtensorMap& tp, const CUtensorMap& tq, const CUtensorMap& tc, const TcParams& prm,
                   cudaStream_t stream) {
    using C = Cfg<BN, kSwap>;
    auto kern = fp8_gemm_tc_kernel<BN, kSwap>;
    static bool configured[64] = {};
    int dev = 0;
    DSV3_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 64 && !configured[dev]) {
        DSV3_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes));
        configured[dev] = true;
    }
    if (prm.cluster) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(static_cast<unsigned>(prm.num_items));
        cfg.blockDim = dim3(kNumThreads);
        cfg.dynamicSmemBytes = C::kSmemBytes;
        cfg.stream = stream;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = static_cast<unsigned>(prm.splits);
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = pdl_enabled() ? 2 : 1;
        DSV3_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, tp, tq, tc, prm));
        return DSV3_OK;
    }
    int grid = prm.num_items < num_sms() ? prm.num_items : num_sms();
    DSV3_CUDA_TRY(launch_dependent(kern, dim3(grid), dim3(kNumThreads), C::kSmemBytes, stream, tp, tq, tc, prm));
    return DSV3_OK;
}

}  // namespace

bool tc_supported(const void* a, const void* b, const void* c, int64_t M, int64_t N, int64_t K) {
    return M > 0 && N > 0 && K >= 16 && (K % 16) == 0 && (reinterpret_cast<uintptr_t>(a) % 16) == 0 &&
           (reinterpret_cast<uintptr_t>(b) % 16) == 0 && (reinterpret_cast<uintptr_t>(c) % 16) == 0 && M < (1ll << 31) && N < (1ll << 31) && K < (1ll << 31);
}

// How many clusters of `splits` CTAs of a variant the device holds at once (GPCs do not divide evenly by every size).
namespace {
thread_local bool t_guessed = false;      // set where the device did not tell
template <int BN, bool kSwap>
int clusters_of(int dev, int splits) {
    using C = Cfg<BN, kSwap>;
    static int cached[64][kMaxClusterSplits + 1] = {};
    if (dev >= 0 && cached[dev][splits] > 0) return cached[dev][splits];
    int n = 0;
    if (dev >= 0) {
        auto kern = fp8_gemm_tc_kernel<BN, kSwap>;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(static_cast<unsigned>(splits));
        cfg.blockDim = dim3(kNumThreads);
        cfg.dynamicSmemBytes = C::kSmemBytes;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = static_cast<unsigned>(splits);
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
            (void)cudaGetLastError();
            n = 0;
        }
        if (n > 0) cached[dev][splits] = n;
    }
    if (n > 0) return n;
    t_guessed = true;
    return 128 / splits;      // no device (planning on a host without one): a cautious guess
}
}  // namespace

static int64_t clusters_resident(int dev, int sms, bool swap, int bn, int splits) {
    const int n = !swap ? (bn == 64 ? clusters_of<64, false>(dev, splits) : clusters_of<128, false>(dev, splits))
                        : (bn == 16 ? clusters_of<16, true>(dev, splits) : (bn == 32 ? clusters_of<32, true>(dev, splits) : clusters_of<64, true>(dev, splits)));
    const int budget = sms / splits;
    return n < budget ? n : budget;
}

// Microseconds of a launch of weight-major tiles of bn tokens, `chunks` K chunks to each of `ctas` CTAs, that HBM does not bound
// (B200, a replayed graph; within 0.4 of 60 shapes of 17 to 256 tokens): set-up, chunks, and for tiles cut over a cluster the exchange,
// which grows with the CTAs that load side by side and, for tiles of 64, with the tokens in them.
static double small_estimate(int bn, int64_t M, int chunks, int splits, int64_t ctas) {
    const double n = static_cast<double>(ctas);
    if (bn == 16) return 2.82 + 0.1875 * chunks + (splits > 1 ? 0.8 + 0.012 * n : 0.0);
    if (bn == 32) return 3.25 + 0.195 * chunks + (splits > 1 ? 0.2 + 0.0155 * n : 0.0);
    if (splits == 1) return 4.1 + 0.28 * chunks;
    const double per_tile = static_cast<double>(M) / static_cast<double>((M + 63) / 64);
    return 3.6 + 0.26 * chunks + 0.6 + 0.0125 * n + (per_tile > 33.0 ? 0.7 * (per_tile - 33.0) / 31.0 : 0.0);
}

// The same of token-major tiles of 64 weight rows (K up to 144 chunks).  Long K lies further from the L2: its chunks take longer; so do those of rows that
// lie multiples of 4 KB apart (N 1536, M 151, two splits: K 4096 8.8 us, K 5120 8.3; M 674, N 1360, K 8192 17.6, K 7680 13.9).
static double half_estimate(int kc, int chunks, int splits, int64_t ctas) {
    const double n = static_cast<double>(ctas), far = (kc <= 56 ? 0.0 : (kc >= 128 ? 0.04 : 0.04 * (kc - 56) / 72.0)) + (kc % 32 ? 0.0 : 0.04);
    return splits == 1 ? 2.97 + (0.18 + far) * chunks + 0.0065 * n : 4.1 + (0.1955 + far) * chunks + 0.0078 * n + 0.123 * (splits - 2);
}

// Time of n wide tiles (256 x 256) on so many pairs, in the plan's microseconds.  The last round may be cut into strips.  Scales that do not
// come four chunks at a time lengthen the chunks, with long rows of them more.  With act_quant, us, tiles of 256 x 256 / 256 x 128: chunks a multiple of
// four, M 4172, N 7168, K 7168 210 / 243; of two, M 3475, N 6432, K 9856 219 / 242, two rounds and long rows, M 1336, N 4624, K 14080 138 / 115; odd, M 1709,
// N 10384, K 5248 104 / 114, a round and a half, M 1418, N 4624, K 7040 69 / 59, strips behind one round, M 1937, N 2944, K 6016 50 / 46.5, long rows, M 5248,
// N 2688, K 14464 286 / 251.
static double wide_estimate(int64_t n, int64_t pairs, int kc) {
    const double more = kc % 4 == 0 ? 1.0 : (kc % 2 ? 1.16 : 1.10) + (kc > 64 ? 0.003 * (kc - 64) : 0.0);
    const int strip = tw_strip_width(n % pairs, pairs, kc);
    if (strip) return 0.5 + static_cast<double>(n / pairs) * (kc * 0.40 * more + 0.9) + kc * (strip == 64 ? 0.30 : 0.39) * more + 1.5;
    return 0.5 + static_cast<double>((n + pairs - 1) / pairs) * (kc * 0.40 * more + 0.9);
}

// Pinned values (dsv3_set_gemm_policy) are honoured or refused (pl.error), never rewritten; the automatic
// plan adapts freely.  dev, sms: the device (-1: none) and the SMs there are on it, or the budget for them.
// estimate: microseconds of an automatic plan of token-major tiles; of others (pl.swap, or anything pinned) it says nothing
static TcPlan work_out_plan(int64_t M, int64_t N, int64_t K, int force_kernel, int force_split, int dev, int sms, double& estimate) {
    TcPlan pl;
    pl.error = DSV3_OK;
    pl.pair = false;
    pl.wide = false;
    pl.splits = 1;
    pl.cluster = false;
    estimate = 0.0;
    pl.kc = static_cast<int>((K + kChunk - 1) / kChunk);
    pl.swap = (force_kernel == 3) || (force_kernel == 0 && M <= 64);
    if (pl.swap) {
        pl.bn = M <= 16 ? 16 : (M <= 32 ? 32 : 64);
        pl.tiles_p = static_cast<int>((N + kPRows - 1) / kPRows);
        pl.tiles_q = static_cast<int>((M + pl.bn - 1) / pl.bn);
    } else {
        pl.bn = 128;
        pl.tiles_p = static_cast<int>((M + kPRows - 1) / kPRows);
        pl.tiles_q = static_cast<int>((N + 127) / 128);
    }
    struct { int bn, tiles_q, splits; } chosen = {0, 0, 0};      // narrower token tiles than these
    double chosen_estimate = 0.0;
    int half_splits = 0;                                         // or token-major tiles of 64 weight rows
    const int64_t tiles = static_cast<int64_t>(pl.tiles_p) * pl.tiles_q;
    if (tiles * 64 >= (1ll << 31)) {     // the work-item counters are 32-bit (at most 64 splits)
        set_last_error("fp8_gemm: %lld output tiles are more than the work-item counter holds", static_cast<long long>(tiles));
        pl.error = DSV3_ERR_UNSUPPORTED;
        return pl;
    }
    int splits = 1;
    const int tab = pl.swap ? scale_tab_chunks(pl.bn) : (1 << 30);   // chunks per item the scale table holds
    if (force_split > 0) {
        splits = force_split;
        const char* why = nullptr;
        if (splits > pl.kc) why = "more splits than 128-wide K chunks";
        else if (splits > 1 && tiles > kMaxTickets) why = "more output tiles than the workspace header has tickets";
        else if ((pl.kc + splits - 1) / splits > tab) why = "K range per split exceeds the weight-major kernel's scale table";
        else if ((force_kernel == 4 || force_kernel == 6) && splits > 1) why = "the CTA-pair kernels do not split K";
        if (why) {
            set_last_error("fp8_gemm: pinned split factor %d cannot be used for M=%lld N=%lld K=%lld: %s", force_split,
                           static_cast<long long>(M), static_cast<long long>(N), static_cast<long long>(K), why);
            pl.error = DSV3_ERR_UNSUPPORTED;
            return pl;
        }
    } else if (force_kernel == 4 || force_kernel == 6) {
        splits = 1;
    } else {
        // Splitting K over the CTAs of a cluster fills idle SMs; every split pays for the exchange of partial tiles.
        // Estimate, fitted to B200 measurements (microseconds; a launch's fixed cost, 2.5-4 us, is left out):
        //   S = 1: rounds * (chunks * c + o)        S > 1 (all clusters resident at once): chunks / S * c + e(S)
        // c = time per K chunk of one CTA; the chunks never take less than the operands need at 6 TB/s, or at 60 GB/s for
        // each CTA there is (weight-major tiles; what a CTA's operand ring can keep in flight).  Measured, us, S = 2 / 3 /
        // 4 / 6 / 8: 12288 -> 5120 at M = 1 15.4 / 13.2 / - / - / -; 7168 -> 2304 at M = 16 9.1 / 8.0 / 7.5 / 6.9 / -; 7168 -> 576
        // at M = 64 11.4 / 9.5 / 8.3 / 7.8 / 7.1; 7168 -> 1536 at M = 200 13.5 / 12.3 / 11.0 / - / -, S = 5 11.3 (rows that do not
        // divide evenly); a split that needs a second round of clusters loses badly (7168 -> 2048 at M = 16, S = 8: 12.9).
        const double c = !pl.swap ? 0.28 : (pl.bn == 64 ? 0.23 : 0.24);
        const double e = !pl.swap ? 4.9 : (pl.bn == 64 ? 1.0 : 0.8), e_split = !pl.swap ? 0.0 : (pl.bn == 64 ? 0.05 : 0.1);
        const double bytes = static_cast<double>(N) * K + static_cast<double>(M) * K;
        const auto hbm_floor = [&](int64_t ctas) { return bytes / (pl.swap && ctas < 100 ? 6.0e4 * ctas : 6.0e6); };
        double best = 1e30;
        if (pl.kc <= tab) {
            best = static_cast<double>((tiles + sms - 1) / sms) * pl.kc * c;
            if (!pl.swap) {
                // Token-major tiles, three kernels: one CTA per 128 x 128 tile, or pairs on 256 x 128 and 256 x 256 tiles.
                // The pairs fold a tile with fewer operand bytes, the small tiles fill the last round better; o = result
                // tile and hand-over, and 0.4 to 1.2 for the cluster launch.  (Chunk times in a full machine; a single round runs at
                // higher clocks.  Chosen so, 277 shapes of 72 to 4000 tokens are within a few per cent of the best of the
                // three; with K below 1536 excluded from the 256 x 128 tiles and no estimate for the single CTA, thirty
                // were 4-39 % away.  949 shapes of 129 to 8000 tokens for which the estimates of the pairs are within a quarter of one another: 0.24 %
                // from the best of the three on average, 3 % of them by more than 3 %.  Estimates too low for wide tiles of odd chunk counts and in strips,
                // and for a single CTA's later rounds (0.37 a chunk of a strip of 128, 0.38 of a tile, 1.12 and 1.05 times as much, 0.29): 0.72 %, and 10 %
                // of them; M 1049, N 4720, K 5504 with act_quant 46.3 / 42.6 us, M 923, N 6464, K 2944 28.8 / 25.3.)
                const int pairs = sms / 2;
                const int64_t pp = (static_cast<int64_t>(pl.tiles_p) + 1) / 2;
                const auto unsplit = [&](int64_t n, int64_t units, double chunk, double chunk1, double o) {
                    const int64_t rounds = (n + units - 1) / units;
                    return static_cast<double>(rounds) * (pl.kc * (rounds == 1 ? chunk1 : chunk) + o);
                };
                best = unsplit(tiles, sms, 0.305, 0.29, 1.0);
                if (force_kernel == 0) {
                    const double full = pp * pl.tiles_q < pairs ? static_cast<double>(pp * pl.tiles_q) / pairs : 1.0;
                    const double pitch = pl.kc % 32 ? 1.0 : 1.1;       // (as in half_estimate())
                    const double narrow = tm_pair_supported(M, N, K) ? pitch * (0.4 + 0.8 * full + unsplit(pp * pl.tiles_q, pairs, 0.265, 0.235, 0.8)) : 1e30;
                    double wide = 1e30;
                    if (tw_pair_supported(M, N, K)) wide = wide_estimate(pp * ((N + 255) / 256), pairs, pl.kc);
                    pl.wide = wide < best && wide <= narrow;
                    pl.pair = pl.wide || narrow < best;
                    if (narrow < best) best = narrow;
                    if (wide < best) best = wide;
                }
            }
            if (const double floor = hbm_floor(tiles); best < floor) best = floor;
        }
        for (int sfac = 2; sfac <= kMaxClusterSplits && sfac <= pl.kc; ++sfac) {
            const int per_item = (pl.kc + sfac - 1) / sfac;
            if (per_item > tab || tiles > clusters_resident(dev, sms, pl.swap, pl.bn, sfac)) continue;
            double t = per_item * c;
            if (const double floor = hbm_floor(tiles * sfac); t < floor) t = floor;
            t += e + e_split * sfac + (!pl.swap && (sfac & (sfac - 1)) ? 0.6 : 0.0);
            if (t < best - 1e-9) {
                best = t;
                splits = sfac;
                pl.cluster = true;
                pl.pair = pl.wide = false;
            }
        }
        // Narrower token tiles.  From 33 to 256 tokens and up to 24 MB of weights a launch is set-up, exchange and a few chunks, and tiles of 16, 32
        // or 64 tokens with the weights on the M side (the weights then come from L2 once per token tile) have less of each: a narrow
        // tile's parts are small, and with enough tiles none is cut.  small_estimate() in absolute microseconds, fitted like the above; the
        // token-major tiles' 2.4 us of launch are added here, and what a cluster loses when many load side by side.
        // us, one tile as wide as M or token-major tiles / so: 7168 -> 576 at M = 33, 64, 128, 256 6.5 / 6.0, 7.2 / 6.3, 9.1 / 7.1, 9.6 / 8.8; 7168 -> 1536 at
        // 64, 96, 192 7.7 / 7.35, 9.8 / 8.7, 10.9 / 10.7; 16384 -> 512 at 64, 128 9.2 / 7.8, 11.25 / 9.0; uncut, 2048 -> 7168 at 64 8.0 / 6.4,
        // 512 -> 4096 at 64, 128 5.3 / 3.7, 5.1 / 4.1, 1536 -> 3072 at 128 7.0 / 5.6, 2048 -> 1408 at 256 7.45 / 6.3.  No gain: 7168 -> 2304 at 33
        // 7.9 / 8.5, 7168 -> 1536 at 256 11.3 / 13.1; with more weights, 16384 -> 7168 at 64 28.5 / 31.7.  (Weights in the L2.  From HBM the gain is smaller, and
        // up to 32 tokens it is a loss: two layers of a decode step, one rank of eight, 32 tokens 303.0 / 307.2, 48 356.3 / 353.2, 64 398.3 / 389.4.)
        double now = best + 2.4 + (pl.cluster ? 0.017 * (static_cast<double>(tiles * splits) - 72.0) : 0.0);
        estimate = now;
        if (force_kernel == 0 && M > 32 && M <= 256 && N * K <= (24ll << 20)) {
            const int64_t rows = (N + kPRows - 1) / kPRows;
            const double margin = pl.swap ? 0.15 : 0.5;     // (what the estimates are apart, of one kernel and of two)
            if (pl.swap) now = tiles * splits <= sms ? small_estimate(pl.bn, M, (pl.kc + splits - 1) / splits, splits, tiles * splits) : 1e30;
            for (int bn = 16; bn <= 64; bn *= 2) {
                const int64_t q = (M + bn - 1) / bn, narrow = rows * q;
                if (pl.swap && bn >= pl.bn) break;
                for (int sfac = 1; sfac <= kMaxClusterSplits && sfac <= pl.kc && narrow * sfac <= sms; ++sfac) {
                    const int per_item = (pl.kc + sfac - 1) / sfac;
                    if (per_item > scale_tab_chunks(bn) || (sfac > 1 && narrow > clusters_resident(dev, sms, true, bn, sfac))) continue;
                    const double t = small_estimate(bn, M, per_item, sfac, narrow * sfac);
                    if (t < now - margin) {
                        now = t + margin;                   // (once, not against one another)
                        chosen = {bn, static_cast<int>(q), sfac};
                        chosen_estimate = t;
                    }
                }
            }
            if (chosen.bn) estimate = now = chosen_estimate;
        }
        // Token-major tiles of 64 weight rows, which never lie in two weight blocks, where they fit one round: a chunk is 24 KB of loads for a CTA
        // instead of 32, a part of a tile half as much to exchange, and there are more ways to come near 148 CTAs.  half_estimate() is
        // fitted to 412 launches of 172 shapes of 70 to 2200 tokens (rms 5 %, weights from HBM, a replayed graph).  Of 520 drawn shapes of 65 to
        // 2200 tokens 176 take them, at 1.13 of the speed of the best of the other kinds by the plan, 1.11 behind act_quant; one is 6 % slower behind it (M 87,
        // N 2240, K 3456 8.4 / 8.9); of 130 that would take narrow token tiles, at 1.10, one 3 %.  us, without them / so: M 1003, N 576, K 7168 12.3 / 10.0; M 256, N 576, K 7168
        // 9.3 / 7.4; M 1000, N 256, K 7168 10.2 / 8.2; M 200, N 2304, K 7168 12.4 / 10.1; M 529, N 1584, K 4224 11.5 / 9.3; M 70, N 7168, K 2304 8.6 / 7.1;
        // M 650, N 800, K 896 5.6 / 4.7.  Clusters of more than two that leave few SMs over wait for room, odd ones, which leave an SM of a pair over, sooner
        // (behind act_quant, M 1328, N 256, K 7168, 44 of three, 15.9 / 18.0; M 1280, 40 of three, 15.7 / 13.4; M 301, N 688, K 7936, 33 of four, 14.0 / 11.2).
        // Beyond 96 MB HBM bounds both (M 107, N 8688, K 14336 28.5 / 30.4).  Against narrow token tiles the estimates, and behind act_quant the
        // launches, are further apart: of 45 shapes with 0.85 between them all but one gain, up to 2.2, of 21 with less seven lose 0.2 to 0.4.
        if (force_kernel == 0 && M > 64 && pl.kc <= 144 && N * K <= (96ll << 20)) {
            const int64_t narrow = static_cast<int64_t>(pl.tiles_p) * ((N + 63) / 64);
            const double margin = chosen.bn ? 0.85 : 0.4;
            for (int sfac = 1; sfac <= kMaxClusterSplits && sfac <= pl.kc && narrow * sfac <= sms; ++sfac) {
                if (sfac > 1 && (narrow > clusters_resident(dev, sms, false, 64, sfac) || (sfac > 2 && 20 * narrow * sfac > (sfac % 2 ? 17 : 18) * sms))) continue;
                const double t = half_estimate(pl.kc, (pl.kc + sfac - 1) / sfac, sfac, narrow * sfac), floor = bytes / 6.0e6 + 2.4;
                if (t < now - margin && floor < now - margin) {
                    now = t + margin;
                    estimate = t;
                    chosen = {0, 0, 0};
                    half_splits = sfac;
                }
            }
        }
    }
    if (half_splits) {
        pl.swap = pl.pair = pl.wide = false;
        pl.bn = 64;
        pl.tiles_p = static_cast<int>((M + kPRows - 1) / kPRows);
        pl.tiles_q = static_cast<int>((N + 63) / 64);
        pl.splits = half_splits;
        pl.cluster = half_splits > 1;
        return pl;
    }
    if (chosen.bn) {
        pl.swap = true;
        pl.pair = pl.wide = false;
        pl.bn = chosen.bn;
        pl.tiles_p = static_cast<int>((N + kPRows - 1) / kPRows);
        pl.tiles_q = chosen.tiles_q;
        pl.splits = chosen.splits;
        pl.cluster = chosen.splits > 1;
        return pl;
    }
    if (force_split == 0 && (pl.kc + splits - 1) / splits > tab) {
        // the weight-major kernel keeps an item's scales in a shared-memory table: split K until an item fits
        splits = (pl.kc + tab - 1) / tab;
        pl.cluster = false;
        if (splits > 32 || tiles > kMaxTickets) {
            if (force_kernel == 3) {
                set_last_error("fp8_gemm: K=%lld is too long for the weight-major kernel's scale table", static_cast<long long>(K));
                pl.error = DSV3_ERR_UNSUPPORTED;
                return pl;
            }
            return work_out_plan(M, N, K, 2, 0, dev, sms, estimate);   // automatic choice, absurdly long K: token-major tiles instead
        }
    }
    pl.splits = splits;
    if (force_kernel == 4 && !tm_pair_supported(M, N, K)) {
        set_last_error("fp8_gemm: the CTA-pair kernel needs more than 128 tokens (M=%lld)", static_cast<long long>(M));
        pl.error = DSV3_ERR_UNSUPPORTED;
        return pl;
    }
    if (force_kernel == 6 && !tw_pair_supported(M, N, K)) {
        set_last_error("fp8_gemm: the 256-wide CTA-pair kernel needs more than 128 tokens and more than 128 weight rows (M=%lld, N=%lld)",
                       static_cast<long long>(M), static_cast<long long>(N));
        pl.error = DSV3_ERR_UNSUPPORTED;
        return pl;
    }
    if (force_kernel == 4 || force_kernel == 6) {
        pl.pair = true;
        pl.wide = force_kernel == 6;
    }
    return pl;
}

// A plan is asked for twice per call, for the workspace and for the launch, and takes 0.1 to 0.2 us to work out, of calls that keep the
// host busy for 4.5: a thread remembers the last sixteen by all that they depend on.  (Looked through in turn, 4 to 15 ns; a slot
// for each by its sizes made the Linears of one layer displace one another.)
static TcPlan planned(int64_t M, int64_t N, int64_t K, int force_kernel, int force_split, double& estimate) {
    int dev = 0;
    const int sms = num_sms_of_device(&dev);
    if (force_kernel != 0 || force_split != 0 || dev < 0) return work_out_plan(M, N, K, force_kernel, force_split, dev, sms, estimate);
    struct Remembered {
        int64_t M, N, K;
        int sms, dev;
        TcPlan plan;
        double estimate;
    };
    constexpr unsigned kRemembered = 16;
    static thread_local Remembered remembered[kRemembered] = {};
    static thread_local unsigned oldest = 0;
    for (const Remembered& r : remembered)
        if (r.M == M && r.N == N && r.K == K && r.sms == sms && r.dev == dev) {
            estimate = r.estimate;
            return r.plan;
        }
    t_guessed = false;
    const TcPlan plan = work_out_plan(M, N, K, 0, 0, dev, sms, estimate);
    if (plan.error == DSV3_OK && !t_guessed) {           // (the message of an error is the call's own)
        remembered[oldest] = {M, N, K, sms, dev, plan, estimate};
        oldest = (oldest + 1) % kRemembered;
    }
    return plan;
}

TcPlan tc_plan(int64_t M, int64_t N, int64_t K, int force_kernel, int force_split) {
    double estimate = 0.0;
    return planned(M, N, K, force_kernel, force_split, estimate);
}

// Whether two weights of one size are multiplied sooner in one launch of wide tiles than in one launch each: the two have one last
// round of the SMs between them instead of one each, and one launch's set-up.  The results are the same bit for bit where both ways
// take tiles that are not cut over K.  B200, us with act_quant, two launches / one: M 2580, N 2304, K 7168 120.9 / 89.5; M 3942, N 2816, K 2048
// 61.4 / 50.2; M 2201, N 2048, K 7168 75.1 / 69.1; M 2201, N 3072, K 5120 93.9 / 68.8; M 500, N 12288, K 5120 91.3 / 66.6; M 8192, N 2048, K 7168
// 266 / 244.  The margin: with many rounds the two are level, or the launch boundary, which brings the pairs back into step,
// is worth 1 %: M 2201, N 18432, K 7168 541 / 551, M 6000, N 12288, K 5120 697 / 704, M 8192, N 18432, K 7168 1917 / 1923.  (Odd numbers of chunks, half
// of it: M 5121, N 2560, K 4992 152 / 148, M 5377, N 4096, K 2944 152 / 148.)
// Not where the common last round would be half full or less (with 24 chunks, or up to a quarter, it would be cut into strips).  The line keeps
// the launches that tests/test_gpu_mlp_launches.py counts, and leaves time there: of 99 such shapes of 11 MLPs two launches are ahead at a dozen, by up
// to 1 %, with many rounds of long rows (M 8191, N 18432, K 7168 1910 / 1917), one launch by up to 40 % at the others: strips, M 2335, N 2304, K 7168
// 111.9 / 87.3, M 1786, N 2816, K 2048 33.8 / 26.3; whole, M 2030, N 2816, K 2048 36.4 / 28.5, M 6910, N 1408, K 2048 59.3 / 49.7.
bool tw_two_pay(int64_t M, int64_t N, int64_t K) {
    if (!tw_pair_supported(M, N, K)) return false;
    double estimate = 0.0;
    const TcPlan one = planned(M, N, K, 0, 0, estimate);
    if (one.error != DSV3_OK || one.swap || estimate <= 0.0) return false;
    const int64_t n = 2 * ((M + 2 * kPRows - 1) / (2 * kPRows)) * ((N + 255) / 256), pairs = num_sms() / 2;
    if (n % pairs != 0 && 2 * (n % pairs) <= pairs) return false;
    double two = wide_estimate(n, pairs, one.kc);
    if (const double floor = (2.0 * static_cast<double>(N) * K + static_cast<double>(M) * K) / 6.0e6; two < floor) two = floor;
    return two + 2.4 < (one.kc % 2 ? 0.98 : 0.975) * 2.0 * estimate;
}

size_t tc_workspace_bytes(const TcPlan& pl, int64_t M, int64_t N) {
    // (A split inside a cluster leaves the workspace untouched; the size is asked for all the same, so that a caller's
    // buffer does not depend on which form a device or an SM budget makes the plan choose.)
    if (pl.splits <= 1) return 0;
    // one padded tile (128 x bn fp32) per (split, tile)
    (void)M;
    (void)N;
    return static_cast<size_t>(DSV3_WORKSPACE_HEADER_BYTES) +
           static_cast<size_t>(pl.splits) * pl.tiles_p * pl.tiles_q * kPRows * pl.bn * sizeof(float);
}

int launch_fp8_gemm_tc(const void* a, const float* a_s, const void* b, const float* b_s, int64_t M, int64_t N,
                       int64_t K, void* c, void* workspace, size_t workspace_bytes, const TcPlan& pl,
                       cudaStream_t stream) {
    if (pl.splits > 1 && !pl.cluster) {
        const size_t need = tc_workspace_bytes(pl, M, N);
        if (!workspace || workspace_bytes < need || (reinterpret_cast<uintptr_t>(workspace) % 256) != 0) {
            set_last_error("fp8_gemm: split-K needs a 256-byte aligned workspace of %zu bytes (got %zu)", need,
                           workspace ? workspace_bytes : static_cast<size_t>(0));
            return DSV3_ERR_WORKSPACE;
        }
    }
    if (pl.error != DSV3_OK) return pl.error;
    // (a plan that overlooks this makes the kernel write past its shared memory; whatever made the plan, it is not launched)
    if (pl.swap && (pl.splits < 1 || (pl.kc + pl.splits - 1) / pl.splits > scale_tab_chunks(pl.bn))) {
        set_last_error("fp8_gemm: %d K chunks in %d parts are more than the weight-major kernel's scale table holds", pl.kc, pl.splits);
        return DSV3_ERR_UNSUPPORTED;
    }
    if (pl.wide) return launch_fp8_gemm_tw(a, a_s, b, b_s, M, N, K, c, stream);
    if (pl.pair) return launch_fp8_gemm_tm(a, a_s, b, b_s, M, N, K, c, stream);
    CUtensorMap tp, tq, tc;
    memset(&tc, 0, sizeof(tc));
    int rc;
    bool tma_store = false;
    if (pl.swap) {
        if ((rc = make_tmap(&tp, b, N, K, kPRows)) != DSV3_OK) return rc;
        if ((rc = make_tmap(&tq, a, M, K, pl.bn)) != DSV3_OK) return rc;
    } else {
        if ((rc = make_tmap(&tp, a, M, K, kPRows)) != DSV3_OK) return rc;
        if ((rc = make_tmap(&tq, b, N, K, pl.bn)) != DSV3_OK) return rc;
        tma_store = pl.bn == 128 && !pl.cluster && (N % 8) == 0;   // row pitch of the result must be a multiple of 16 bytes for a tensor map
        if (tma_store && (rc = make_tmap_out(&tc, c, M, N)) != DSV3_OK) return rc;
    }
    TcParams prm;
    prm.a_s = a_s;
    prm.b_s = b_s;
    prm.c = static_cast<__nv_bfloat16*>(c);
    prm.tickets = static_cast<int*>(workspace);
    prm.partials = workspace ? reinterpret_cast<float*>(static_cast<uint8_t*>(workspace) + DSV3_WORKSPACE_HEADER_BYTES)
                             : nullptr;
    prm.status = status_device_ptr();
    if (!prm.status) return DSV3_ERR_CUDA;
    prm.M = M;
    prm.N = N;
    prm.kc = pl.kc;
    prm.tiles_p = pl.tiles_p;
    prm.tiles_q = pl.tiles_q;
    prm.splits = pl.splits;
    prm.cluster = pl.cluster ? 1 : 0;
    prm.tma_store = tma_store ? 1 : 0;
    // Work order: `raster` token tiles share consecutive weight tiles.  For token-major tiles the group is
    // made as tall as keeps its activations (raster x 128 x K bytes) within about a quarter of L2, so that
    // the weights are streamed from HBM as few times as possible.
    prm.raster = 8;
    if (!pl.swap) {
        const int64_t fit = (32ll << 20) / (static_cast<int64_t>(kPRows) * K);
        prm.raster = static_cast<int>(fit < 8 ? 8 : (fit > 64 ? 64 : fit));
    }
    prm.div_rows = make_fast_div(static_cast<uint32_t>((kPRows + pl.splits - 1) / pl.splits));
    prm.div_splits = make_fast_div(static_cast<uint32_t>(prm.splits));
    prm.div_raster = make_fast_div(static_cast<uint32_t>(prm.raster));
    prm.div_per_group = make_fast_div(static_cast<uint32_t>(prm.raster) * static_cast<uint32_t>(prm.tiles_q));
    prm.num_items = pl.tiles_p * pl.tiles_q * pl.splits;   // < 2^31: checked by tc_plan
    if (pl.swap) {
        switch (pl.bn) {
            case 16: return launch_variant<16, true>(tp, tq, tc, prm, stream);
            case 32: return launch_variant<32, true>(tp, tq, tc, prm, stream);
            case 64: return launch_variant<64, true>(tp, tq, tc, prm, stream);
        }
    } else if (pl.bn == 128) {
        return launch_variant<128, false>(tp, tq, tc, prm, stream);
    } else if (pl.bn == 64) {
        return launch_variant<64, false>(tp, tq, tc, prm, stream);
    }
    set_last_error("fp8_gemm: no tcgen05 variant for tile width %d", pl.bn);
    return DSV3_ERR_UNSUPPORTED;
}

// ---------------------------------------------------------------------------------------------
// Self-test of what the tcgen05 kernels do when a wait gives up: one warp waits, with the given limit, for an mbarrier
// phase that nothing will ever complete, while seven others already stand in the barrier that the eight share.  The wait
// runs out, records (kind 9, counter, CTA) in the status words, and the warp takes part in the barrier with what it knows;
// every warp turns away and the kernel returns normally: nothing traps, faults or spins without a bound.  (A warp that
// the barrier told otherwise records kind 10.)
// ---------------------------------------------------------------------------------------------
namespace {

__global__ void bounded_wait_selftest_kernel(unsigned int* status, uint64_t limit_ns) {
    __shared__ uint64_t bar;
    __shared__ Control ctl;
    if (threadIdx.x == 0) {
        ctl.abort_flag = 0;
        mbar_init(smem_u32(&bar), 1);
        mbar_fence_init();
    }
    __syncthreads();
    bool ok = true;
    if (threadIdx.x < 32) ok = __all_sync(0xffffffffu, bounded_wait_ns(smem_u32(&bar), 0, &ctl, status, 9, 0, limit_ns));
    if (barrier_all<256>(1, ok)) status[1] = 10;
}

}  // namespace

int launch_bounded_wait_selftest(uint64_t limit_ns, cudaStream_t stream) {
    unsigned int* status = status_device_ptr();
    if (!status) return DSV3_ERR_CUDA;
    bounded_wait_selftest_kernel<<<1, 256, 0, stream>>>(status, limit_ns);
    DSV3_CUDA_TRY(cudaGetLastError());
    return DSV3_OK;
}

}  // namespace dsv3
