// Weight-streaming FP8 GEMM for sm_100a: few tokens per weight, every weight byte read once.  Used for the expert
// loop of an expert layer (all local experts, and for few rows the shared experts, in one launch per projection) and, without
// groups, for w1 and w3 of an MLP whose tiles fit one round (swiglu_linear_tile); w1 and w3 carry SwiGLU and the quantisation in
// front of w2 in their epilogue.
//
// Replaces the per-expert act_quant + fp8_gemm calls of MoE.forward, inference/model.py:683-689 and :633, and
// `F.silu(w1(x)) * w3(x)` followed by w2's act_quant, model.py:532 and :158-159.
//
// What bounds it: HBM.  An SM's share of the copy bandwidth is 43 GB/s, one 32 KB pair of weight blocks per 0.75 us.
//   * A tile is TWO 128-row weight blocks (rows 128 j.. of w1 and of w3; or two neighbouring blocks of one weight)
//     against up to BN tokens: the token tile crosses from L2 once per 256 weight rows instead of once per 128, and
//     both halves of a SwiGLU pair meet in the same thread's registers.
//   * Up to 64 tokens per tile: weights are the M operand (128 TMEM lanes), tokens the N operand, and a tile of 16 tokens
//     costs 16 columns (stream_tiles).  Up to 128 tokens: tokens are the M operand (rows_tiles).  With many tokens
//     one launch has CTAs of both, each for the groups that suit it (stream_tile).
//   * Uneven split: where whole tiles would leave the last round of SMs mostly idle, the (tile, K chunk) space is cut into
//     equal contiguous ranges, one per CTA (struct Plan).  A CTA then has at most two partial tiles (the head
//     and the tail of its range); they are parked as fp32 (valid tokens only) and the CTA that takes a tile's last ticket
//     adds them in K order, so the result does not depend on timing and nothing spins.
//
// Roles: warp 0 TMA producer, warp 1 MMA issuer (both converged, one elected lane issues), warps 4..11 promotion: every
// chunk product leaves TMEM and is folded into fp32 registers with its two scales (kernel.py:162).
//
// Every mbarrier wait is bounded (tc_wait.cuh); producers wait for the last commits onto their barriers before the
// CTA leaves.  A promotion warp whose wait gave up goes on through the tiles without working on them, to take part in the
// barriers where other warps may be waiting for it (barrier_all).
#include <cuda.h>

#include <cstring>
#include <vector>

#include "common.cuh"
#include "gemm_plan.cuh"
#include "quant_math.cuh"
#include "tc_wait.cuh"

namespace dsv3 {

namespace {

constexpr int kNumThreads = 384;
constexpr int kFirstPromoWarp = 4;
constexpr int kPromoThreads = 256;
constexpr int kTabThreads = 64;
constexpr int kRegsControl = 40;
constexpr int kRegsPromo = 232;
static_assert(128 * kRegsControl + 256 * kRegsPromo <= 384 * 168, "register pool");
// weights on the M side: fewer accumulators; the control warps' tile bookkeeping does not fit 40 registers (a spilled
// variable goes through an L1 that the operand stages have squeezed out: 5 % of an expert layer)
constexpr int kRegsControlM = 88;
constexpr int kRegsPromoM = 208;
static_assert(128 * kRegsControlM + 256 * kRegsPromoM <= 384 * 168, "register pool");
constexpr int kMaxGroups = kMaxGroupsOfTable;

// kRows: tokens on the M side (rows_tiles); otherwise weights (stream_tiles).
template <int BN_, bool kRows>
struct SCfg {
    static constexpr int BN = BN_;
    static constexpr int kBox = BN < 32 ? BN : 32;                    // token rows per TMA box
    static constexpr int kTokBytes = BN * kChunk;
    static constexpr int kStageBytes = kTokBytes + 2 * kPRows * kChunk;   // tokens and two weight blocks of one chunk
    static constexpr int kStages = BN <= 32 ? 6 : (BN <= 64 ? 5 : 4);
    static constexpr int kSlotCols = kRows ? 2 * kPRows : 2 * BN;     // TMEM columns of one chunk product
    static constexpr int kSlots = kRows ? 2 : (BN <= 32 ? 8 : 512 / kSlotCols);
    static constexpr int kTmemCols = kSlots * kSlotCols;
    // weights on the M side: ring of scales, per-warp maxima and final scales
    static constexpr int kTabChunks = BN <= 16 ? 16 : (BN <= 32 ? 12 : 8);              // K chunks per slot of the scale ring
    static constexpr int kTabBytes = kRows ? 0 : 2 * kTabChunks * 2 * BN * 4;         // token scale x block scale, of both blocks
    static constexpr int kSegBytes = kRows ? 0 : (kMaxGroups + 1) * 4;           // row offsets of the groups
    static constexpr int kRedBytes = kRows ? 0 : (4 + 1) * BN * 4;
    // tokens on the M side: exchange of SwiGLU halves / staging of results
    static constexpr int kXBytes = kRows ? 2 * BN * 128 : 0;
    // barriers, control words, group prefix and scan
    static constexpr int kCtlBytes = (2 * kStages + 2 * kSlots + 4) * 8 + static_cast<int>(sizeof(Control)) + (kMaxGroups + 1 + 8) * 4;
    static constexpr int kSmemBytes = 1024 + kStages * kStageBytes + kTabBytes + kRedBytes + kXBytes + kCtlBytes + kSegBytes;
    static_assert(kStageBytes >= kPRows * kChunk + kTokBytes || !kRows, "the MMA's 128 token rows stay inside the stage");
    static_assert(kSmemBytes <= 232448, "shared memory per CTA");
    static_assert(kSmemBytes > 116 * 1024, "one CTA per SM");
    static_assert(kTmemCols >= 32 && kTmemCols <= 512 && (kTmemCols & (kTmemCols - 1)) == 0, "TMEM columns");
};

// A launch works on up to two problems that share the shape of a tile: the groups (per-group weights, rows by group) and
// one ordinary weight (the shared experts next to the routed ones; kBoth).
struct Side {
    int kc, nblk, tiles_p;              // K chunks, 128-row blocks of a weight, tiles per token tile
    int rows;                           // rows of a (ordinary weight)
    const float* a_s;                   // token scales: a_s[row * as_row + chunk * as_chunk]
    int64_t as_row, as_chunk;
    __nv_bfloat16* c;                   // plain: bf16 [rows, N]
    int64_t N;
    int vec_store;                      // rows of c are 16-byte aligned
    uint8_t* hq;                        // SwiGLU: e4m3 [rows, N]
    float* hs;                          // SwiGLU: hs[row * hs_row + block * hs_blk]
    int64_t hs_row, hs_blk;
};
constexpr int kGroups = 0, kOrdinary = 1;
struct StreamParams {
    Side side[2];
    // groups: block b of a tile comes from map / scale set b, in global memory; row offsets seg[n_groups + 1] likewise
    const CUtensorMap* g_map[2];
    const float* const* g_scale[2];
    const int* seg;
    int n_groups;
    int min_rows, max_rows;             // groups with fewer or more rows are not this problem's
    int first_cta, ctas;                // the CTAs of the grid that work on it
    uint64_t coprime;                   // bit i: i has no factor in common with ctas
    const float* scale[2];              // ordinary weight (its maps are kernel parameters)
    int scale_fmt;
    int leads, early;                   // StreamGemm::leads, early
    // split tiles
    float* partials;                    // [CTA][2][2 * BN / 4][128] float4, or null: whole tiles only
    int* tickets;                       // one per CTA, zero on entry and on exit
    unsigned int* status;
};

struct Seg {          // a range of K chunks of one tile
    int side, kc, ut; // which problem, its K chunks, the tile's first unit
    int c0, c1;
    int row0, ntok;   // token rows
    int group, p;     // weight, tile within the weight
};

// The CTA's share of the work; every CTA derives the same plan from the same numbers.  The tiles (the groups' first, then
// the ordinary weight's) are worked on whole, one after the other per CTA, or (kSplit) where that would leave the machine
// idle in the last of one or two rounds, the (tile, K chunk) space is cut into equal contiguous ranges, one per CTA.
// Whole tiles of the ordinary weight are spread among the groups': the ordinary weight is read once and multiplied by
// many tokens, so its tiles keep the tensor core busy and HBM idle while the groups' do the opposite, and side by side on
// different SMs they share the machine.  Their distance has no factor in common with the number of CTAs, or they would all be
// the same few CTAs'.  us per layer in a replayed graph, ordinary weight last / spread: 32 of 256 experts of 7168 x 2048 with the shared
// one, 200 tokens 228.7 / 213.2, 333 256.9 / 228.1, 512 299.5 / 263.5; 160 of 5120 x 1536 with two, 512 658 / 626; 64 of 2048 x 1408 with
// two, 333 tokens 133.2 / 128.7, 1024 188 / 186.  Where the groups have fewer than twice as many tiles, and the CTAs are even in number,
// the only such distance is 1: the ordinary weight comes first.  So 16 of 64 experts of 2048 x 1408, 2048 tokens (352 and 352 tiles) 125.5
// last, 123.8 first, 126.4 at a distance of 3 with the rest at the end; 32 of 256 of 7168 x 2048, 1800 and 2048 398.6, 394.4, 401.2 and
// 420.2, 411.4, 422.2; 64 of 2048 x 1408, 512 (231 and 88) 143.9, 143.6, 143.7; 32 of those, 600 (143 and 110) 97.4, 97.5, 96.5.
// Where the ordinary weight has more tiles than the groups they stay last (8 of 64 experts of 2048 x 1408, 512
// tokens: 59.8 last, 62.2 first): the groups' tiles wait for HBM and are better begun early.  Short ones (less than half the groups' K:
// w2 of a tensor-parallel shard of the shared expert) stay last as well, where they fill up the last round: two layers of a decode
// step, one rank of eight, at 16, 32 and 64 tokens 236.2 / 308.1 / 404.7 spread, 234.1 / 305.9 / 401.1 last.
// (Cutting only the tiles of the last round was slower: each then has about ten parts, which one CTA adds up while the
// others wait for it.  So was cutting a problem of more rounds: 14 rounds of 40 chunks took 380 us whole, 476 cut.)
// A unit is one K chunk of a tile.  32-bit arithmetic throughout (the host checks that the units fit): a 64-bit division
// takes about half a microsecond here, and ranges computed as units * cta / ctas cost a small problem 15 us.
struct Plan {
    int kc0, kc1;            // K chunks: groups, ordinary weight
    int tiles0, tiles1;      // groups, ordinary weight
    int every;               // whole tiles: every so-manieth is one of the ordinary weight while there are any (1: they come first; 0: last)
    int G;                   // CTAs that take a range
    int units, base, extra;  // the first `extra` CTAs take base + 1 units, the others base
    __device__ __forceinline__ int begin(int cta) const { return cta * base + min(cta, extra); }
    __device__ __forceinline__ int owner(int u) const {
        const int head = extra * (base + 1);
        return u < head ? static_cast<int>(static_cast<unsigned>(u) / static_cast<unsigned>(base + 1))
                        : extra + static_cast<int>(static_cast<unsigned>(u - head) / static_cast<unsigned>(base));
    }
};

// group_tiles: token tiles over all groups
template <int BN, bool kBoth, bool kSplit>
__device__ __forceinline__ Plan make_plan(const StreamParams& p, int group_tiles) {
    Plan pl;
    pl.tiles0 = p.side[kGroups].tiles_p * group_tiles;
    pl.tiles1 = kBoth ? p.side[kOrdinary].tiles_p * ((p.side[kOrdinary].rows + BN - 1) / BN) : 0;
    pl.kc0 = p.side[kGroups].kc;
    pl.kc1 = p.side[kOrdinary].kc;
    pl.units = pl.tiles0 * pl.kc0 + pl.tiles1 * pl.kc1;
    pl.G = pl.base = pl.extra = 0;
    pl.every = 0;
    const int ctas = p.ctas;
    if constexpr (kBoth && !kSplit) {
        if (pl.tiles1 > 0 && pl.tiles0 >= pl.tiles1 && 2 * pl.kc1 >= pl.kc0) {
            // (the distances that will do come from the host: looking for one here, by division, cost 0.6 us)
            const int most = min(63, static_cast<int>(static_cast<unsigned>(pl.tiles0 + pl.tiles1) / static_cast<unsigned>(pl.tiles1)));
            pl.every = 63 - __clzll(static_cast<long long>(p.coprime & (~0ull >> (63 - most))));
        }
    }
    const int rounds = static_cast<int>(static_cast<unsigned>(pl.tiles0) / static_cast<unsigned>(ctas));
    const int rest0 = pl.tiles0 - rounds * ctas;
    if constexpr (!kSplit) return pl;
    if (rounds < 2) {
        const int G = cut_ranges(BN, pl.tiles0 + pl.tiles1, pl.units, rest0 * pl.kc0 + pl.tiles1 * pl.kc1,
                                 max(rest0 > 0 ? pl.kc0 : 0, pl.tiles1 > 0 ? pl.kc1 : 0), ctas);
        if (G > 0) {
            pl.G = G;
            pl.base = static_cast<int>(static_cast<unsigned>(pl.units) / static_cast<unsigned>(G));
            pl.extra = pl.units - pl.base * G;
        }
    }
    return pl;
}

// Iterates over the segments of a CTA.
template <int BN, bool kBoth, bool kSplit>
struct Walker {
    const StreamParams& p;
    const Plan& pl;
    const int* prefix;       // shared memory: token tiles of the groups before each group
    const int* seg;          // row offsets of the groups, in shared memory, or where a tile is long enough in global
    int u, u1;               // next unit and end of the CTA's range
    int tile;                // next whole tile
    __device__ __forceinline__ Walker(const StreamParams& p_, const Plan& pl_, const int* prefix_, const int* seg_) : p(p_), pl(pl_), prefix(prefix_), seg(seg_) {
        const int cta = static_cast<int>(blockIdx.x) - p.first_cta;
        u = kSplit && cta < pl.G ? pl.begin(cta) : 0;
        u1 = kSplit && cta < pl.G ? pl.begin(cta + 1) : 0;
        tile = cta;
    }
    __device__ __forceinline__ bool next(Seg& s) {
        int at;                  // tile within the side
        if (kSplit && u < u1) {
            const int units0 = pl.tiles0 * pl.kc0;
            s.side = !kBoth || u < units0 ? kGroups : kOrdinary;
            s.kc = (!kBoth || s.side == kGroups) ? pl.kc0 : pl.kc1;
            const int v = (!kBoth || s.side == kGroups) ? u : u - units0;
            at = static_cast<int>(static_cast<unsigned>(v) / static_cast<unsigned>(s.kc));
            s.ut = u - v + at * s.kc;
            s.c0 = u - s.ut;
            s.c1 = min(s.kc, s.c0 + (u1 - u));
            u += s.c1 - s.c0;
        } else {
            if ((kSplit && pl.G > 0) || tile >= pl.tiles0 + pl.tiles1) return false;
            if (kBoth && !kSplit && pl.every > 0) {
                const int j = static_cast<int>(static_cast<unsigned>(tile) / static_cast<unsigned>(pl.every));
                s.side = j < pl.tiles1 && j * pl.every == tile ? kOrdinary : kGroups;
                at = s.side == kOrdinary ? j : tile - min(pl.tiles1, j + 1);
            } else {
                s.side = !kBoth || tile < pl.tiles0 ? kGroups : kOrdinary;
                at = (!kBoth || s.side == kGroups) ? tile : tile - pl.tiles0;
            }
            s.kc = (!kBoth || s.side == kGroups) ? pl.kc0 : pl.kc1;
            s.ut = 0;
            s.c0 = 0;
            s.c1 = s.kc;
            tile += p.ctas;
        }
        // inside a weight the token tile runs fastest, so CTAs that work side by side share the weight blocks
        int nq, first, rows;
        if (!kBoth || s.side == kGroups) {
            const int per = p.side[kGroups].tiles_p;
            int lo = 0, hi = p.n_groups;
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (prefix[mid] * per <= at) lo = mid; else hi = mid;
            }
            s.group = lo;
            nq = prefix[lo + 1] - prefix[lo];
            at -= prefix[lo] * per;
            first = BN == 128 ? __ldcg(seg + lo) : seg[lo];
            rows = (BN == 128 ? __ldcg(seg + lo + 1) : seg[lo + 1]) - first;
        } else {
            s.group = 0;
            rows = p.side[kOrdinary].rows;
            nq = (rows + BN - 1) / BN;
            first = 0;
        }
        s.p = nq == 1 ? at : at / nq;
        const int q = at - s.p * nq;
        s.row0 = first + q * BN;
        s.ntok = min(BN, rows - q * BN);
        return true;
    }
};

// Token tiles per group and their exclusive prefix sum over the groups, into shared memory (all threads of the CTA;
// the caller synchronises before prefix[] is read).
template <int BN>
__device__ __forceinline__ void prefix_groups(const StreamParams& p, int* prefix, int* scan, int* seg, int warp, int lane) {
    int v = 0;
    if (threadIdx.x < kMaxGroups) {
        const int e = threadIdx.x;
        if (e < p.n_groups) {
            const int first = __ldcg(p.seg + e), end = __ldcg(p.seg + e + 1);
            const int rows = end - first;
            v = rows >= p.min_rows && rows <= p.max_rows ? (rows + BN - 1) / BN : 0;
            if (seg) {
                seg[e] = first;
                if (e == p.n_groups - 1) seg[e + 1] = end;
            }
        }
        int inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) scan[warp] = inc;
        v = inc - v;
    }
    __syncthreads();
    if (threadIdx.x < kMaxGroups) {
        for (int w = 0; w < warp; ++w) v += scan[w];
        prefix[threadIdx.x] = v;
    }
    if (threadIdx.x == 0) {
        int tot = 0;
        for (int w = 0; w < kMaxGroups / 32; ++w) tot += scan[w];
        prefix[kMaxGroups] = tot;        // groups beyond n_groups hold no tiles
    }
}

// The groups' tensor maps and scale pointers on their way from HBM into the L2, where a CTA's first loads would otherwise wait for
// them: the weights of the layers in between have long displaced them.  Each CTA asks for a few lines, while what comes before
// this kernel is still running (the tables do not change; the L2 is the point of coherence).  us per layer in a replayed graph, without /
// with: 64 experts of 2048 x 1408, 16 and 333 tokens 78.2 / 78.0, 125.7 / 125.4; 32 of 256 of 7168 x 2048, 16 112.3 / 112.1.
__device__ __forceinline__ void prefetch_tables(const StreamParams& p, int lane, int warp) {
    if (warp != 3) return;
    const int lines = p.n_groups + (p.n_groups * 8 + 127) / 128;
    for (int i = static_cast<int>(blockIdx.x) - p.first_cta + lane * p.ctas; i < lines; i += 32 * p.ctas)
#pragma unroll
        for (int b = 0; b < 2; ++b) asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const uint8_t*>(p.g_map[b]) + i * 128));
}

// The TMA producer (one converged warp).  Stage: [BN token rows][block 0][block 1] of one K chunk; of the tokens only
// the boxes that hold any of the tile's rows are fetched.  With `early` the kernel before this one may still be running: the first
// weights are fetched all the same, the tokens, which it writes, behind the wait for it.
template <class C, bool kSwiglu, bool kBoth, bool kSplit>
__device__ __forceinline__ void produce(const StreamParams& p, const Plan& pl, const int* prefix, const int* seg, const void* w0, const void* w1,
                                        const void* ta0, const void* ta1, uint32_t tiles, uint32_t bar0, Control* ctl) {
    constexpr int NS = C::kStages, BN = C::BN;
    Walker<BN, kBoth, kSplit> wk(p, pl, prefix, seg);
    Seg s;
    uint32_t g = 0;
    bool ok = true, early = p.early != 0;
    while (ok && wk.next(s)) {
        const void* m0 = (!kBoth || s.side == kGroups) ? static_cast<const void*>(p.g_map[0] + s.group) : w0;
        const void* m1 = (!kBoth || s.side == kGroups) ? static_cast<const void*>(p.g_map[1] + s.group) : w1;
        const void* ta = (!kBoth || s.side == kGroups) ? ta0 : ta1;
        const int r0 = (kSwiglu ? s.p : 2 * s.p) * kPRows;
        const int r1 = kSwiglu ? r0 : r0 + kPRows;
        const bool two = kSwiglu || 2 * s.p + 1 < p.side[kBoth ? s.side : kGroups].nblk;
        const int boxes = (s.ntok + C::kBox - 1) / C::kBox;
        const uint32_t bytes = (two ? 2u : 1u) * kPRows * kChunk + static_cast<uint32_t>(boxes) * C::kBox * kChunk;
        int k = s.c0;
        if (early) {
            early = false;
            const int n = min(NS, s.c1 - s.c0);
            if (elect_one()) {
                for (int i = 0; i < n; ++i) {
                    const uint32_t full = bar0 + 8u * i, dst = tiles + i * C::kStageBytes;
                    mbar_arrive_expect_tx(full, bytes);
                    tma_load_2d(dst + C::kTokBytes, m0, (k + i) * kChunk, r0, full);
                    if (two) tma_load_2d(dst + C::kTokBytes + kPRows * kChunk, m1, (k + i) * kChunk, r1, full);
                }
            }
            __syncwarp();
            griddep_wait();
            if (elect_one()) {
                for (int i = 0; i < n; ++i)
                    for (int b = 0; b < boxes; ++b)
                        tma_load_2d(tiles + i * C::kStageBytes + b * C::kBox * kChunk, ta, (k + i) * kChunk, s.row0 + b * C::kBox, bar0 + 8u * i);
            }
            __syncwarp();
            k += n;
            g = n;
        }
        for (; k < s.c1; ++k, ++g) {
            const int st = g % NS;
            const uint32_t full = bar0 + 8u * st, empty = bar0 + 8u * (NS + st);
            ok = __all_sync(0xffffffffu, bounded_wait(empty, ((g / NS) & 1u) ^ 1u, ctl, p.status, 1, g));
            if (!ok) break;
            if (elect_one()) {
                const uint32_t dst = tiles + st * C::kStageBytes;
                mbar_arrive_expect_tx(full, bytes);
                tma_load_2d(dst + C::kTokBytes, m0, k * kChunk, r0, full);
                if (two) tma_load_2d(dst + C::kTokBytes + kPRows * kChunk, m1, k * kChunk, r1, full);
                for (int b = 0; b < boxes; ++b) tma_load_2d(dst + b * C::kBox * kChunk, ta, k * kChunk, s.row0 + b * C::kBox, full);
            }
            __syncwarp();
        }
    }
    if (early) griddep_wait();                 // (no work)
    // nothing else waits for the commits onto the empty[] barriers of the last chunks: none may be in flight
    // when the CTA leaves (it would land in whatever CTA gets this shared memory next)
    for (uint32_t d = (g > static_cast<uint32_t>(NS) ? g - NS : 0u); ok && d < g; ++d)
        ok = __all_sync(0xffffffffu, bounded_wait(bar0 + 8u * (NS + d % NS), (d / NS) & 1u, ctl, p.status, 1, d));
}

// Ticket of a partial tile whose parts are parked (promotion threads): whether this CTA holds the tile's last ticket.
// ok comes in as "this warp's waits have succeeded" and goes out as "every warp's have"; without that no ticket is taken.
__device__ __forceinline__ bool last_part(const StreamParams& p, Control* ctl, int first, int last, bool& ok) {
    ok = barrier_all<256>(1, ok);
    if (!ok) return false;
    if (threadIdx.x == kFirstPromoWarp * 32) {
        int tk;
        // releases the parked tile (cumulative over the barrier) and acquires the other parts
        asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(tk) : "l"(p.tickets + first) : "memory");
        if (tk == last - first) p.tickets[first] = 0;
        ctl->ticket[0] = tk;
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");
    const bool mine = ctl->ticket[0] == last - first;
    asm volatile("bar.sync 1, 256;" ::: "memory");            // the slot may be overwritten from here on
    return mine;
}

__device__ __forceinline__ void teardown(Control* ctl, int warp, uint32_t tmem_base, uint32_t cols) {
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (ctl->abort_flag) {
        // give copies and MMAs that were already issued time to land before shared memory and TMEM are released
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        tc_dealloc(tmem_base, cols);
    }
}

// ---------------------------------------------------------------------------------------------------------------------
// Weights on the M side (128 TMEM lanes), the tile's tokens on the N side: an MMA's N is the number of tokens rounded up
// to 16, so neither the tensor core nor the promotion warps work on token slots that are empty.  (With tokens on the M
// side the same expert layer, 57 tokens per tile, drew the board's whole power at 1380 MHz: half of the multiplications
// were for nobody.)  Promotion group g owns every second piece of 16 tokens, of both blocks.
// ---------------------------------------------------------------------------------------------------------------------
template <int BN, bool kSwiglu, bool kBoth, bool kSplit>
__device__ __forceinline__ void stream_tiles(const CUtensorMap* tmap_w0, const CUtensorMap* tmap_w1, const CUtensorMap* tmap_a0, const CUtensorMap* tmap_a1,
                                             const StreamParams& p) {
    using C = SCfg<BN, false>;
    constexpr int NS = C::kStages, NT = C::kSlots, TC = C::kTabChunks;
    constexpr int PW = BN == 16 ? 8 : 16;  // tokens per piece
    constexpr int NP = BN / 2 / PW;        // pieces per promotion thread: piece i covers tokens (2 i + group) PW ...

    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t tiles = (raw + 1023u) & ~1023u;
    uint8_t* gen = smem_raw + (tiles - raw);
    float* tab = reinterpret_cast<float*>(gen + NS * C::kStageBytes);                 // [2][TC][2][BN] token scale x scale of block 0, 1
    float* red = reinterpret_cast<float*>(gen + NS * C::kStageBytes + C::kTabBytes);  // [4][BN] maxima, then [BN] scales
    uint64_t* bars = reinterpret_cast<uint64_t*>(gen + NS * C::kStageBytes + C::kTabBytes + C::kRedBytes);
    Control* ctl = reinterpret_cast<Control*>(bars + 2 * NS + 2 * NT + 4);
    int* prefix = reinterpret_cast<int*>(ctl + 1);
    int* scan = prefix + kMaxGroups + 1;                                              // [8] warp totals
    int* seg = scan + 8;                                                              // [kMaxGroups + 1]
    const uint32_t bar0 = smem_u32(bars);
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (NS + s); };
    auto tfull_bar = [&](int s) { return bar0 + 8u * (2 * NS + s); };
    auto tempty_bar = [&](int s) { return bar0 + 8u * (2 * NS + NT + s); };
    auto sfull_bar = [&](int s) { return bar0 + 8u * (2 * NS + 2 * NT + s); };        // slot of the scale ring is filled
    auto sempty_bar = [&](int s) { return bar0 + 8u * (2 * NS + 2 * NT + 2 + s); };

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int s = 0; s < NT; ++s) {
            mbar_init(tfull_bar(s), 1);
            mbar_init(tempty_bar(s), kPromoThreads / 32);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(sfull_bar(s), kTabThreads);
            mbar_init(sempty_bar(s), kPromoThreads / 32);
        }
        ctl->abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(tmap_a0);
        if constexpr (kBoth) {
            tma_prefetch_desc(tmap_a1);
            tma_prefetch_desc(tmap_w0);
            tma_prefetch_desc(tmap_w1);
        }
    }
    if (warp == 1) tc_alloc(smem_u32(&ctl->tmem_base), C::kTmemCols);
    if (!p.leads) griddep_launch_dependents();
    prefetch_tables(p, lane, warp);
    if (!p.early) griddep_wait();
    if (p.leads) griddep_launch_dependents();  // behind the wait: what an early dependent relies on
    prefix_groups<BN>(p, prefix, scan, seg, warp, lane);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = ctl->tmem_base;
    const Plan pl = make_plan<BN, kBoth, kSplit>(p, prefix[kMaxGroups]);

    if (p.early && warp != 0) griddep_wait();  // (the producer: behind its first weights)
    if (warp < kFirstPromoWarp) {
      if constexpr (NP >= 2) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsControlM));
      if (warp == 0) {
        produce<C, kSwiglu, kBoth, kSplit>(p, pl, prefix, seg, tmap_w0, tmap_w1, tmap_a0, tmap_a1, tiles, bar0, ctl);
      } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        Walker<BN, kBoth, kSplit> wk(p, pl, prefix, seg);
        Seg s;
        uint32_t g = 0;
        bool ok = true;
        while (ok && wk.next(s)) {
            const bool two = kSwiglu || 2 * s.p + 1 < p.side[kBoth ? s.side : kGroups].nblk;
            const uint32_t idesc = umma_idesc_e4m3_f32(kPRows, 16) + ((static_cast<uint32_t>(s.ntok + 15) / 16 - 1) << 18);   // N in units of 8 at bit 17
            for (int k = s.c0; k < s.c1; ++k, ++g) {
                const int st = g % NS, ts = g % NT;
                ok = __all_sync(0xffffffffu, bounded_wait(tempty_bar(ts), ((g / NT) & 1u) ^ 1u, ctl, p.status, 3, g) &&
                                             bounded_wait(full_bar(st), (g / NS) & 1u, ctl, p.status, 2, g));
                if (!ok) break;
                tc_fence_after();
                const uint32_t sp = tiles + st * C::kStageBytes;
                const uint64_t dt = umma_desc_k_major_sw128(sp);
                const uint64_t d0 = umma_desc_k_major_sw128(sp + C::kTokBytes);
                const uint64_t d1 = umma_desc_k_major_sw128(sp + C::kTokBytes + kPRows * kChunk);
                const uint32_t d_tmem = tmem_base + ts * C::kSlotCols;
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < kChunk / 32; ++kk) tc_mma_f8(d_tmem, d0 + 2u * kk, dt + 2u * kk, idesc, kk > 0 ? 1u : 0u);
                    if (two) {
#pragma unroll
                        for (int kk = 0; kk < kChunk / 32; ++kk)
                            tc_mma_f8(d_tmem + BN, d1 + 2u * kk, dt + 2u * kk, idesc, kk > 0 ? 1u : 0u);
                    }
                    tc_commit(empty_bar(st));
                    tc_commit(tfull_bar(ts));
                }
                __syncwarp();
            }
        }
      } else {
        // ------------------------------------------------------------ scales, TC chunks at a time
        Walker<BN, kBoth, kSplit> wk(p, pl, prefix, seg);
        Seg s;
        uint32_t t = 0;          // ring counter
        bool ok = true;
        const int tid = threadIdx.x - 64;
        // Block scales: a lane loads that of block lane % 2 of chunk lane / 2 and the warp's lanes hand them round (with a load of
        // its own for each of a thread's products, three for one, 64-token tiles took up to 6 % longer, cut ones of 16 and 32 up
        // to 2 %).  Whole tiles of 16 and 32 are ahead by up to 1 % with loads of their own.  us, own loads / handed round, one
        // layer: 64-token tiles, 256 experts of 7168 x 2048 at 1003 tokens 1937 / 1823, 160 of 5120 x 1536 at 700 680 / 644;
        // divided, 1600 tokens 870 / 829; cut, 20 of 160 of 5120 x 1536 at 12 tokens 50.6 / 49.5; whole 32-token
        // tiles, 32 of 256 of 7168 x 2048 at 280 tokens 251.8 / 253.7.
        constexpr bool kOwn = BN > 32 || kSplit;
        while (ok && wk.next(s)) {
            const Side& d = p.side[kBoth ? s.side : kGroups];
            auto block_scales = [&](int b) {
                const int blk = kSwiglu ? s.p : min(2 * s.p + b, d.nblk - 1);
                return ((!kBoth || s.side == kGroups) ? p.g_scale[b][s.group] : p.scale[b]) + static_cast<int64_t>(blk) * s.kc;
            };
            const float* bs0 = block_scales(kOwn ? lane & 1 : 0);
            [[maybe_unused]] const float* bs1 = kOwn ? nullptr : block_scales(1);
            for (int k = s.c0; k < s.c1; k += TC, ++t) {
                const int sl = t & 1;
                ok = __all_sync(0xffffffffu, bounded_wait(sempty_bar(sl), ((t >> 1) & 1u) ^ 1u, ctl, p.status, 7, t));
                if (!ok) break;
                const int n = min(TC, s.c1 - k);
                float* dst = tab + sl * TC * 2 * BN;
                // All loads of a slot are in flight together: they queue behind the weights' (one after the other they held
                // the first chunk back by 7 us).  Columns beyond ntok keep what they held: they multiply products nobody reads.
                constexpr int kLoads = TC * BN / kTabThreads;
                static_assert(kTabThreads % BN == 0 || BN % kTabThreads == 0, "a thread's columns do not depend on the trip");
                static_assert(2 * TC <= 32, "one block scale per lane");
                float r[kLoads], rb[kLoads][2], own = 0.0f;
                if (kOwn && (lane >> 1) < n) own = __ldg(bs0 + k + (lane >> 1));
#pragma unroll
                for (int u = 0; u < kLoads; ++u) {
                    const int i = tid + u * kTabThreads, ch = i / BN, col = i - ch * BN;
                    if (ch < n && col < s.ntok) {
                        r[u] = __ldg(d.a_s + (s.row0 + col) * d.as_row + (k + ch) * d.as_chunk);
                        if constexpr (!kOwn) {
                            rb[u][0] = __ldg(bs0 + k + ch);
                            rb[u][1] = __ldg(bs1 + k + ch);
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < kLoads; ++u) {
                    const int i = tid + u * kTabThreads, ch = i / BN, col = i - ch * BN;
                    if constexpr (kOwn) {
                        rb[u][0] = __shfl_sync(0xffffffffu, own, 2 * ch);
                        rb[u][1] = __shfl_sync(0xffffffffu, own, 2 * ch + 1);
                    }
                    if (ch < n && col < s.ntok) {
                        dst[ch * 2 * BN + col] = r[u] * rb[u][0];
                        dst[ch * 2 * BN + BN + col] = r[u] * rb[u][1];
                    }
                }
                mbar_arrive(sfull_bar(sl));
            }
        }
      }
    } else {
        if constexpr (NP >= 2) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsPromoM));
        // ------------------------------------------------------------ promotion + epilogue
        const int grp = (warp - kFirstPromoWarp) >> 2;
        const int col0 = grp * PW;
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;                    // weight row within a block (TMEM lane)
        const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + col0;
        auto kc_of = [&](const Seg& q) { return kBoth ? q.kc : p.side[kGroups].kc; };
        Walker<BN, kBoth, kSplit> wk(p, pl, prefix, seg);
        Seg s;
        uint32_t g = 0, t = 0;
        bool ok = true;
        float2 acc[2][NP][PW / 2];
        uint32_t v[NP > 1 ? 2 : 1][2][PW];
        auto load_piece = [&](uint32_t taddr, int i, uint32_t (&vv)[2][PW]) {
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                if constexpr (PW == 8) tc_ld_x8(taddr + b * BN + 2 * PW * i, vv[b]);
                else tc_ld_x16(taddr + b * BN + 2 * PW * i, vv[b]);
            }
        };
        // acc += product * (a_s * b_s), the order of the other tcgen05 kernels, so that a tile that is not cut equals theirs bit
        // for bit.  The scale warps form a_s * b_s once per CTA: formed here, by every thread for all of its rows, the
        // multiplications took as much of the FP32 pipes as the sums (64-token tiles, 256 experts of 7168 x 2048 with 64 tokens
        // each: 2936 -> 2724 us).
        auto fold_piece = [&](const float* as, int i, const uint32_t (&vv)[2][PW]) {
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const float4* as4 = reinterpret_cast<const float4*>(as + b * BN + 2 * PW * i);
#pragma unroll
                for (int j = 0; j < PW / 4; ++j) {
                    const float4 a4 = as4[j];
                    acc[b][i][2 * j] = __ffma2_rn(make_float2(__uint_as_float(vv[b][4 * j]), __uint_as_float(vv[b][4 * j + 1])), make_float2(a4.x, a4.y), acc[b][i][2 * j]);
                    acc[b][i][2 * j + 1] = __ffma2_rn(make_float2(__uint_as_float(vv[b][4 * j + 2]), __uint_as_float(vv[b][4 * j + 3])), make_float2(a4.z, a4.w), acc[b][i][2 * j + 1]);
                }
            }
        };
        while (wk.next(s)) {
            const Side& d = p.side[kBoth ? s.side : kGroups];
            // pieces of this thread that hold a token of the tile
            const int np = s.ntok <= col0 ? 0 : min(NP, (s.ntok - col0 + 2 * PW - 1) / (2 * PW));
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int i = 0; i < NP; ++i)
#pragma unroll
                    for (int j = 0; j < PW / 2; ++j) acc[b][i][j] = make_float2(0.0f, 0.0f);
            int in_tab = 0;                         // chunk within the slot of the scale ring
            const int n_ch = s.c1 - s.c0;
            for (int k = 0; ok && k < n_ch; ++k, ++g) {
                const int sl = t & 1;
                if (in_tab == 0) {
                    ok = __all_sync(0xffffffffu, bounded_wait_lean(sfull_bar(sl), (t >> 1) & 1u, ctl, p.status, 8, t));
                    if (!ok) break;
                }
                const float* as = tab + (sl * TC + in_tab) * 2 * BN + col0;
                const int ts = g % NT;
                ok = __all_sync(0xffffffffu, bounded_wait_lean(tfull_bar(ts), (g / NT) & 1u, ctl, p.status, 4, g));
                if (!ok) break;
                tc_fence_after();
                const uint32_t taddr = t_lane + ts * C::kSlotCols;
                auto release = [&] {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(tempty_bar(ts));
                };
                if (np > 0) load_piece(taddr, 0, v[0]);
                if constexpr (NP > 1) {
                    if (np > 1) load_piece(taddr, 1, v[1]);
                }
                tc_wait_ld();
                if (NP <= 2 || np <= 2) release();
                if (np > 0) fold_piece(as, 0, v[0]);
                if constexpr (NP > 1) {
                    if (np > 1) fold_piece(as, 1, v[1]);
                }
                if constexpr (NP > 2) {
                    if (np > 2) {
                        load_piece(taddr, 2, v[0]);
                        if (np > 3) load_piece(taddr, 3, v[1]);
                        tc_wait_ld();
                        release();
                        fold_piece(as, 2, v[0]);
                        if (np > 3) fold_piece(as, 3, v[1]);
                    }
                }
                if (++in_tab == TC || k == n_ch - 1) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(sempty_bar(sl));
                    in_tab = 0;
                    ++t;
                }
            }
            if (!kSplit && !kSwiglu && !ok) break; // (no barrier ahead)

            if (kSplit && n_ch < kc_of(s)) {
                // part of a tile: park the pieces that hold tokens, take a ticket; the last part of the tile adds all
                // parts in K order and goes on to write the result
                const int cta = static_cast<int>(blockIdx.x) - p.first_cta;
                const int first = pl.owner(s.ut), last = pl.owner(s.ut + kc_of(s) - 1);
                constexpr int kTileVec = 2 * BN / 4 * kPRows;             // float4 per parked tile: [2 blocks][BN / 4][128 rows]
                float4* base = reinterpret_cast<float4*>(p.partials) + (col0 / 4) * kPRows + row;
                auto part = [&](int c) { return base + (static_cast<int64_t>(c) * 2 + (pl.begin(c) >= s.ut ? 0 : 1)) * kTileVec; };
                if (ok) {
                    float4* dst = part(cta);
#pragma unroll
                    for (int i = 0; i < NP; ++i)
                        if (i < np)
#pragma unroll
                            for (int b = 0; b < 2; ++b)
#pragma unroll
                                for (int j = 0; j < PW / 4; ++j)
                                    __stcg(dst + (b * (BN / 4) + i * (PW / 2) + j) * kPRows,
                                           make_float4(acc[b][i][2 * j].x, acc[b][i][2 * j].y, acc[b][i][2 * j + 1].x, acc[b][i][2 * j + 1].y));
                }
                const bool mine = last_part(p, ctl, first, last, ok);
                if (!ok) break;                    // all eight warps
                if (!mine) continue;
#pragma unroll
                for (int i = 0; i < NP; ++i) {
                    if (i >= np) continue;
#pragma unroll
                    for (int b = 0; b < 2; ++b)
#pragma unroll
                        for (int j = 0; j < PW / 2; ++j) acc[b][i][j] = make_float2(0.0f, 0.0f);
                    // four parts in flight: one after the other, each costs an L2 round trip (0.5 us), and a tile of a
                    // small problem has up to twenty parts
                    for (int c0 = first; c0 <= last; c0 += 4) {
                        float4 f[4][2][PW / 4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const float4* src = part(min(c0 + u, last));
#pragma unroll
                            for (int b = 0; b < 2; ++b)
#pragma unroll
                                for (int j = 0; j < PW / 4; ++j) f[u][b][j] = __ldcg(src + (b * (BN / 4) + i * (PW / 2) + j) * kPRows);
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            if (c0 + u > last) break;
#pragma unroll
                            for (int b = 0; b < 2; ++b)
#pragma unroll
                                for (int j = 0; j < PW / 4; ++j) {
                                    acc[b][i][2 * j] = __fadd2_rn(acc[b][i][2 * j], make_float2(f[u][b][j].x, f[u][b][j].y));
                                    acc[b][i][2 * j + 1] = __fadd2_rn(acc[b][i][2 * j + 1], make_float2(f[u][b][j].z, f[u][b][j].w));
                                }
                        }
                    }
                }
            }
            if constexpr (!kSwiglu) {
                if (!ok) continue;
                if (BN == 64 && d.vec_store) {
                    // A thread holds one column; four neighbours exchange four tokens so that each stores four columns of one, and a warp
                    // four tokens' 64 bytes at a time.  A store takes the SM 8 cycles with one token's and 13 with four: a tile of 64 tokens 3800
                    // / 2500 cycles of 21000 (us, w2 of 64 experts of 7168 x 2048, 64 rows each 178 / 167, 2048 x 1408 48.8 / 45.2; layers of 32
                    // of 256 experts at 2206 tokens 469.5 / 462.1, 16 of 64 small ones at 600 70.8 / 70.0).  With few tokens the exchange only
                    // lengthens the chain: 16 tokens 800 / 950, 8 of 64 small experts at 62 tokens (tiles of 32) 37.2 / 38.1.
                    const int odd = lane & 1, up = (lane >> 1) & 1;
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        const int64_t n = static_cast<int64_t>(2 * s.p + b) * kPRows + (row & ~3);
                        if ((2 * s.p + b) * kPRows + quarter * 32 >= d.N) continue;        // uniform in the warp
                        __nv_bfloat16* out = d.c + (static_cast<int64_t>(s.row0) + col0 + odd + 2 * up) * d.N + n;
#pragma unroll
                        for (int i = 0; i < NP; ++i) {
                            if (i >= np) continue;
#pragma unroll
                            for (int j = 0; j < PW; j += 4) {
                                const uint32_t w0 = pack_bf16x2(acc[b][i][j / 2].x, acc[b][i][j / 2].y), w1 = pack_bf16x2(acc[b][i][j / 2 + 1].x, acc[b][i][j / 2 + 1].y);
                                const uint32_t p0 = __shfl_xor_sync(0xffffffffu, w0, 1), p1 = __shfl_xor_sync(0xffffffffu, w1, 1);
                                // tokens j + odd and j + 2 + odd of two columns
                                const uint32_t a0 = odd ? __byte_perm(p0, w0, 0x7632) : __byte_perm(w0, p0, 0x5410);
                                const uint32_t a1 = odd ? __byte_perm(p1, w1, 0x7632) : __byte_perm(w1, p1, 0x5410);
                                const uint32_t r = __shfl_xor_sync(0xffffffffu, up ? a0 : a1, 2);
                                if (col0 + 2 * PW * i + j + odd + 2 * up < s.ntok && n < d.N)
                                    *reinterpret_cast<uint2*>(out + (2 * PW * i + j) * d.N) = up ? make_uint2(r, a1) : make_uint2(a0, r);
                            }
                        }
                    }
                    continue;
                }
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const int64_t n = static_cast<int64_t>(2 * s.p + b) * kPRows + row;
                    if (n < d.N) {
                        __nv_bfloat16* out = d.c + (static_cast<int64_t>(s.row0) + col0) * d.N + n;
#pragma unroll
                        for (int i = 0; i < NP; ++i) {
                            if (i >= np) continue;
#pragma unroll
                            for (int j = 0; j < PW; ++j)
                                if (col0 + 2 * PW * i + j < s.ntok)
                                    out[(2 * PW * i + j) * d.N] = __float2bfloat16_rn(j & 1 ? acc[b][i][j / 2].y : acc[b][i][j / 2].x);
                        }
                    }
                }
            } else {
                // h1 and h3 as bf16 (as the operators would have written them), two tokens to a word; then
                // h = bf16(bf16(silu(h1)) * h3) for eight tokens at a time and act_quant over the tile's 128 columns of
                // every token: the maximum is taken across the lanes of a warp and, through shared memory, across the
                // group's warps.  The loops are rolled over registers that turn by one group per trip (unrolled, the
                // epilogue outgrows the instruction cache).
                constexpr int NG = NP * PW / 8;                            // groups of eight tokens
                uint32_t h1[4 * NG], h3[4 * NG];
#pragma unroll
                for (int i = 0; i < NP; ++i)
#pragma unroll
                    for (int j = 0; j < PW / 2; ++j) {
                        h1[i * (PW / 2) + j] = pack_bf16x2(acc[0][i][j].x, acc[0][i][j].y);
                        h3[i * (PW / 2) + j] = pack_bf16x2(acc[1][i][j].x, acc[1][i][j].y);
                    }
                // first token of group q
                auto token = [&](int q) { return PW == 8 ? col0 : col0 + 2 * PW * (q >> 1) + 8 * (q & 1); };
#pragma unroll 1
                for (int q = 0; ok && q < NG; ++q) {
                    const int tk = token(q), rem = s.ntok - tk;
                    uint32_t h[4] = {0u, 0u, 0u, 0u};
                    if (rem > 0) {
                        uint32_t mask[4];                                  // slots beyond the tile's tokens hold anything
#pragma unroll
                        for (int e = 0; e < 4; ++e) mask[e] = 2 * e + 1 < rem ? 0xFFFFFFFFu : (2 * e < rem ? 0xFFFFu : 0u);
                        const uint4 r = swiglu8(make_uint4(h1[0] & mask[0], h1[1] & mask[1], h1[2] & mask[2], h1[3] & mask[3]),
                                                make_uint4(h3[0] & mask[0], h3[1] & mask[1], h3[2] & mask[2], h3[3] & mask[3]));
                        h[0] = r.x; h[1] = r.y; h[2] = r.z; h[3] = r.w;
                        uint32_t top = 0u;
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const uint32_t a = (e & 1 ? h[e / 2] >> 16 : h[e / 2]) & 0x7FFFu;
                            const uint32_t m = __reduce_max_sync(0xffffffffu, a > 0x7F80u ? 0u : a);   // (a NaN is dropped, as in act_quant)
                            if (lane == e) top = m;
                        }
                        if (lane < 8) red[quarter * BN + tk + lane] = __uint_as_float(top << 16);
                    }
#pragma unroll
                    for (int e = 0; e < 4 * NG - 4; ++e) {
                        h1[e] = h1[e + 4];
                        h3[e] = h3[e + 4];
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) h1[4 * NG - 4 + e] = h[e];
                }
                ok = barrier_all<128>(2 + grp, ok);
                if (!ok) {                         // this group's four warps; the barrier of a partial tile counts them too
                    if constexpr (kSplit) continue;
                    else break;
                }
                {
                    const int gt = threadIdx.x & 127;
                    const int tk = col0 + 2 * PW * (gt / PW) + gt % PW;
                    if (gt < NP * PW && tk < s.ntok) {
                        const float m = fmaxf(fmaxf(red[tk], red[BN + tk]), fmaxf(red[2 * BN + tk], red[3 * BN + tk]));
                        const float sc = scale_from_amax(m, p.scale_fmt);
                        red[4 * BN + tk] = rcp_approx(sc);
                        d.hs[(static_cast<int64_t>(s.row0) + tk) * d.hs_row + s.p * d.hs_blk] = sc;
                    }
                }
                asm volatile("bar.sync %0, 128;" ::"r"(2 + grp) : "memory");
                uint8_t* out = d.hq + static_cast<int64_t>(s.row0) * d.N + static_cast<int64_t>(s.p) * kPRows + row;
#pragma unroll 1
                for (int q = 0; q < NG; ++q) {
                    const int tk = token(q), rem = s.ntok - tk;
                    if (rem > 0) {
                        const float* sc = red + 4 * BN + tk;
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float lo = bf16_bits_to_float(h1[e] & 0xFFFFu), hi = __uint_as_float(h1[e] & 0xFFFF0000u);
                            const float s0 = sc[2 * e], s1 = sc[2 * e + 1];
                            const uint32_t two8 = cvt_e4m3x2(__fmul_rn(lo, s0), __fmul_rn(hi, s1));
                            if (2 * e < rem) out[(tk + 2 * e) * d.N] = static_cast<uint8_t>(two8 & 0xFFu);
                            if (2 * e + 1 < rem) out[(tk + 2 * e + 1) * d.N] = static_cast<uint8_t>(two8 >> 8);
                        }
                    }
#pragma unroll
                    for (int e = 0; e < 4 * NG - 4; ++e) h1[e] = h1[e + 4];
                }
                // the next tile's maxima must not overtake this tile's scales
                asm volatile("bar.sync %0, 128;" ::"r"(2 + grp) : "memory");
            }
        }
    }
    teardown(ctl, warp, tmem_base, C::kTmemCols);
}

// ---------------------------------------------------------------------------------------------------------------------
// Up to 128 tokens per tile: tokens on the M side (128 TMEM lanes), the two weight blocks side by side on the N side.
//
// With weights on the M side a token's scale varies along a thread's registers (a shared-memory load per four tokens and
// block) and a token's maximum spans 128 threads.  Here a thread owns one token row and 128
// columns of one block: one scale product per chunk and thread, and a row's maximum is two threads' business.  The MMA
// costs 512 cycles per chunk whatever the number of tokens, which the weights' arrival (1300 cycles at 1.85 GHz) hides.
// ---------------------------------------------------------------------------------------------------------------------
template <int BN, bool kSwiglu, bool kBoth>
__device__ __forceinline__ void rows_tiles(const CUtensorMap* tmap_w0, const CUtensorMap* tmap_w1, const CUtensorMap* tmap_a0, const CUtensorMap* tmap_a1,
                                           const CUtensorMap* tmap_c0, const CUtensorMap* tmap_c1, const StreamParams& p) {
    using C = SCfg<BN, true>;
    constexpr bool kSplit = false;      // its partial tiles would be 128 KB each
    constexpr int NS = C::kStages, NT = C::kSlots;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t tiles = (raw + 1023u) & ~1023u;
    uint8_t* gen = smem_raw + (tiles - raw);
    uint8_t* xbuf = gen + NS * C::kStageBytes;                                 // [2][BN][128 bytes]
    uint64_t* bars = reinterpret_cast<uint64_t*>(xbuf + C::kXBytes);
    Control* ctl = reinterpret_cast<Control*>(bars + 2 * NS + 2 * NT);
    int* prefix = reinterpret_cast<int*>(ctl + 1);
    int* scan = prefix + kMaxGroups + 1;
    const uint32_t bar0 = smem_u32(bars);
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (NS + s); };
    auto tfull_bar = [&](int s) { return bar0 + 8u * (2 * NS + s); };
    auto tempty_bar = [&](int s) { return bar0 + 8u * (2 * NS + NT + s); };

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int s = 0; s < NT; ++s) {
            mbar_init(tfull_bar(s), 1);
            mbar_init(tempty_bar(s), kPromoThreads / 32);
        }
        ctl->abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(tmap_a0);
        if constexpr (kBoth) {
            tma_prefetch_desc(tmap_a1);
            tma_prefetch_desc(tmap_w0);
            tma_prefetch_desc(tmap_w1);
        }
    }
    if (warp == 1) tc_alloc(smem_u32(&ctl->tmem_base), C::kTmemCols);
    if (!p.leads) griddep_launch_dependents();
    prefetch_tables(p, lane, warp);
    if (!p.early) griddep_wait();
    if (p.leads) griddep_launch_dependents();  // behind the wait: what an early dependent relies on
    prefix_groups<BN>(p, prefix, scan, static_cast<int*>(nullptr), warp, lane);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = ctl->tmem_base;
    const Plan pl = make_plan<BN, kBoth, kSplit>(p, prefix[kMaxGroups]);

    if (p.early && warp != 0) griddep_wait();  // (the producer: behind its first weights)
    if (warp < kFirstPromoWarp) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsControl));
        if (warp == 0) {
            produce<C, kSwiglu, kBoth, kSplit>(p, pl, prefix, p.seg, tmap_w0, tmap_w1, tmap_a0, tmap_a1, tiles, bar0, ctl);
        } else if (warp == 1) {
            // -------------------------------------------------------- MMA issuer
            Walker<BN, kBoth, kSplit> wk(p, pl, prefix, p.seg);
            Seg s;
            uint32_t g = 0;
            bool ok = true;
            while (ok && wk.next(s)) {
                const bool two = kSwiglu || 2 * s.p + 1 < p.side[kBoth ? s.side : kGroups].nblk;
                const uint32_t idesc = two ? umma_idesc_e4m3_f32(kPRows, 2 * kPRows) : umma_idesc_e4m3_f32(kPRows, kPRows);
                for (int k = s.c0; k < s.c1; ++k, ++g) {
                    const int st = g % NS, ts = g % NT;
                    ok = __all_sync(0xffffffffu, bounded_wait(tempty_bar(ts), ((g / NT) & 1u) ^ 1u, ctl, p.status, 3, g) &&
                                                 bounded_wait(full_bar(st), (g / NS) & 1u, ctl, p.status, 2, g));
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t sp = tiles + st * C::kStageBytes;
                    // 128 token rows are multiplied; the rows beyond the tile's lie in the weight blocks behind the
                    // tokens (still inside the stage) and produce lanes that nobody reads
                    const uint64_t da = umma_desc_k_major_sw128(sp);
                    const uint64_t db = umma_desc_k_major_sw128(sp + C::kTokBytes);
                    const uint32_t d_tmem = tmem_base + ts * 256;
                    if (elect_one()) {
#pragma unroll
                        for (int kk = 0; kk < kChunk / 32; ++kk) tc_mma_f8(d_tmem, da + 2u * kk, db + 2u * kk, idesc, kk > 0 ? 1u : 0u);
                        tc_commit(empty_bar(st));
                        tc_commit(tfull_bar(ts));
                    }
                    __syncwarp();
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsPromo));
        // ------------------------------------------------------------ promotion + epilogue
        const int grp = (warp - kFirstPromoWarp) >> 2;          // weight block
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;                    // token row of the tile (TMEM lane)
        const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + grp * kPRows;
        uint8_t* my_x = xbuf + grp * (BN * 128);                // this group's half of the exchange buffer
        uint8_t* other_x = xbuf + (1 - grp) * (BN * 128);
        auto kc_of = [&](const Seg& q) { return kBoth ? q.kc : p.side[kGroups].kc; };
        Walker<BN, kBoth, kSplit> wk(p, pl, prefix, p.seg);
        Seg s, ahead;
        uint32_t g = 0;
        bool ok = true;
        float2 acc[64];
        uint32_t v[64];
        auto fold = [&](float sc, int off) {
            const float2 sc2 = make_float2(sc, sc);
#pragma unroll
            for (int j = 0; j < 32; ++j)
                acc[off + j] = __ffma2_rn(make_float2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])), sc2, acc[off + j]);
        };
        auto release = [&](int ts) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty_bar(ts));
        };
        // Scales of this row for four chunks are in flight or in registers, each register re-used for the chunk four
        // further on: a chunk takes 0.3 us to fold, a load that misses L1 about
        // 0.6 us, and with one chunk of look-ahead every chunk waited for it (1330 cycles instead of 700).  A tile's
        // first scales are requested before the result of the tile before it is written.
        const float *as = nullptr, *bs = nullptr;
        int64_t as_chunk = 0;
        float ra[4], rb;         // rb: the weight block's scale of the next chunk (32 chunks to a cache line: L1)
        auto scales_of = [&](const Seg& q) {
            const int blk = kSwiglu ? q.p : 2 * q.p + grp;
            const Side& d = p.side[kBoth ? q.side : kGroups];
            as_chunk = d.as_chunk;
            as = d.a_s + (q.row0 + min(row, q.ntok - 1)) * d.as_row + q.c0 * as_chunk;
            bs = ((!kBoth || q.side == kGroups) ? p.g_scale[grp][q.group] : p.scale[grp]) + static_cast<int64_t>(min(blk, d.nblk - 1)) * kc_of(q) + q.c0;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int k = min(i, q.c1 - q.c0 - 1);
                ra[i] = __ldg(as + k * as_chunk);
            }
            rb = __ldg(bs);
        };
        bool more = wk.next(ahead);
        if (more) scales_of(ahead);
        while (more) {
            s = ahead;
            const Side& d = p.side[kBoth ? s.side : kGroups];
            const int blk = kSwiglu ? s.p : 2 * s.p + grp;
            const bool active = quarter * 32 < s.ntok && blk < d.nblk;     // uniform in the warp
            const int n_ch = s.c1 - s.c0;
#pragma unroll
            for (int j = 0; j < 64; ++j) acc[j] = make_float2(0.0f, 0.0f);
            for (int k0 = 0; ok && k0 < n_ch; k0 += 4) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int k = k0 + i;
                    if (!ok || k >= n_ch) break;
                    const int ts = g % NT;
                    ok = __all_sync(0xffffffffu, bounded_wait_lean(tfull_bar(ts), (g / NT) & 1u, ctl, p.status, 4, g));
                    ++g;
                    if (!ok) break;
                    tc_fence_after();
                    if (!active) {
                        release(ts);
                        continue;
                    }
                    const uint32_t taddr = t_lane + ts * 256;
                    tc_ld_x64(taddr, v);
                    const float sc = ra[i] * rb;
                    ra[i] = __ldg(as + min(k + 4, n_ch - 1) * as_chunk);
                    rb = __ldg(bs + min(k + 1, n_ch - 1));
                    tc_wait_ld();
                    fold(sc, 0);
                    tc_ld_x64(taddr + 64, v);
                    tc_wait_ld();
                    release(ts);
                    fold(sc, 32);
                }
            }
            if (!kSwiglu && !ok) break;            // (no barrier ahead)
            more = wk.next(ahead);
            if (more) scales_of(ahead);

            if (quarter * 32 >= s.ntok) continue;
            if constexpr (!kSwiglu) {
                if (!active) continue;
                // 32 rows x 64 columns at a time through the warp's own 4 KB; where all of the rows are the tile's, from there by a TMA
                // store (an SM's stores go out at 25 bytes per clock, 2600 cycles for a tile, which nobody then waits for).  us, w2 of 32 experts of
                // 7168 x 2048 with 512 rows each 332 / 316, 64 of 2048 x 1408 with 128 and 512 44.1 / 41.9, 128 / 119.
                uint8_t* wbuf = my_x + quarter * (32 * 128);
                const int64_t n0 = static_cast<int64_t>(blk) * kPRows;
                const bool whole = d.vec_store && quarter * 32 + 32 <= s.ntok;
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    if (lane == 0) bulk_wait_group_read0();        // the store before has read the buffer
                    __syncwarp();
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const float2* a = acc + half * 32 + c * 4;
                        *reinterpret_cast<uint4*>(wbuf + lane * 128 + ((c ^ (lane & 7)) << 4)) =
                            make_uint4(pack_bf16x2(a[0].x, a[0].y), pack_bf16x2(a[1].x, a[1].y), pack_bf16x2(a[2].x, a[2].y), pack_bf16x2(a[3].x, a[3].y));
                    }
                    if (whole) {
                        fence_proxy_async_shared();
                        __syncwarp();
                        if (lane == 0) {
                            tma_store_2d(!kBoth || s.side == kGroups ? tmap_c0 : tmap_c1, smem_u32(wbuf), static_cast<int>(n0) + half * 64, s.row0 + quarter * 32);
                            bulk_commit_group();
                        }
                        continue;
                    }
                    __syncwarp();
                    const int piece = lane & 7;
                    const int64_t n = n0 + half * 64 + piece * 8;
#pragma unroll
                    for (int r0 = 0; r0 < 32; r0 += 4) {
                        const int r = r0 + (lane >> 3);
                        if (quarter * 32 + r >= s.ntok) continue;
                        const uint4 o = *reinterpret_cast<const uint4*>(wbuf + r * 128 + ((piece ^ (r & 7)) << 4));
                        __nv_bfloat16* dst = d.c + (static_cast<int64_t>(s.row0) + quarter * 32 + r) * d.N + n;
                        if (d.vec_store && n + 8 <= d.N) {
                            *reinterpret_cast<uint4*>(dst) = o;
                        } else {
                            const uint32_t w4[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
                            for (int e = 0; e < 8; ++e)
                                if (n + e < d.N) reinterpret_cast<uint16_t*>(dst)[e] = static_cast<uint16_t>(w4[e >> 1] >> (16 * (e & 1)));
                        }
                    }
                }
            } else {
                // h1 of a row sits in one group's thread, h3 in the other's: each gives the other half of its columns
                // (bf16, as the operators would have written them) and computes h = bf16(bf16(silu(h1)) * h3) for the 64
                // columns it keeps.  The two threads' maxima meet in the exchange slots they have just read.
                const int give = 1 - grp;                                  // column half handed over
                const uint32_t slot = static_cast<uint32_t>(row) * 128;
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const float2* a = acc + c * 4;
                    const float2* b = acc + 32 + c * 4;
                    const uint4 lo = make_uint4(pack_bf16x2(a[0].x, a[0].y), pack_bf16x2(a[1].x, a[1].y), pack_bf16x2(a[2].x, a[2].y), pack_bf16x2(a[3].x, a[3].y));
                    const uint4 hi = make_uint4(pack_bf16x2(b[0].x, b[0].y), pack_bf16x2(b[1].x, b[1].y), pack_bf16x2(b[2].x, b[2].y), pack_bf16x2(b[3].x, b[3].y));
                    *reinterpret_cast<uint4*>(my_x + slot + ((c ^ (row & 7)) << 4)) = give ? hi : lo;
                    v[4 * c] = give ? lo.x : hi.x;
                    v[4 * c + 1] = give ? lo.y : hi.y;
                    v[4 * c + 2] = give ? lo.z : hi.z;
                    v[4 * c + 3] = give ? lo.w : hi.w;
                }
                ok = barrier_all<64>(2 + quarter, ok);
                if (!ok) break;                    // both warps of these rows
                float m = 0.0f;
                // Rolled loops over a register file that turns by one group per trip: unrolled, this epilogue was longer
                // than the instruction cache holds and cost 8000-14000 cycles per tile.  (Rows beyond the tile's hold
                // products of weights with weights, which nobody reads.)
                if (row < s.ntok) {
#pragma unroll 1
                    for (int c = 0; c < 8; ++c) {
                        const uint4 mine = make_uint4(v[0], v[1], v[2], v[3]);
                        const uint4 theirs = *reinterpret_cast<const uint4*>(other_x + slot + ((c ^ (row & 7)) << 4));
                        const uint4 h = grp == 0 ? swiglu8(mine, theirs) : swiglu8(theirs, mine);
#pragma unroll
                        for (int e = 0; e < 28; ++e) v[e] = v[e + 4];
                        v[28] = h.x;
                        v[29] = h.y;
                        v[30] = h.z;
                        v[31] = h.w;
                        m = fmaxf(m, amax8(h));
                    }
                }
                // only this thread reads slot `row` of the other group's half
                *reinterpret_cast<float*>(other_x + slot) = m;
                asm volatile("bar.sync %0, 64;" ::"r"(2 + quarter) : "memory");
                m = fmaxf(m, *reinterpret_cast<const float*>(my_x + slot));
                if (row < s.ntok) {
                    const float scale = scale_from_amax(m, p.scale_fmt), r = rcp_approx(scale);
                    const int64_t tok = static_cast<int64_t>(s.row0) + row;
                    if (grp == 0) d.hs[tok * d.hs_row + s.p * d.hs_blk] = scale;
                    uint4* out = reinterpret_cast<uint4*>(d.hq + tok * d.N + static_cast<int64_t>(s.p) * kPRows + grp * 64);
#pragma unroll 1
                    for (int c = 0; c < 4; ++c) {
                        const uint4 a = make_uint4(v[0], v[1], v[2], v[3]);
                        const uint4 b = make_uint4(v[4], v[5], v[6], v[7]);
#pragma unroll
                        for (int e = 0; e < 24; ++e) v[e] = v[e + 8];
                        const uint2 qa = quant8(a, r), qb = quant8(b, r);
                        out[c] = make_uint4(qa.x, qa.y, qb.x, qb.y);
                    }
                }
            }
        }
    }
    if (!kSwiglu && warp >= kFirstPromoWarp && lane == 0) bulk_wait_group0();      // results have left shared memory
    teardown(ctl, warp, tmem_base, C::kTmemCols);
}

template <int BN, bool kSwiglu, bool kBoth, bool kSplit>
__global__ void __launch_bounds__(kNumThreads, 1)
fp8_stream_kernel(const __grid_constant__ CUtensorMap tmap_w0, const __grid_constant__ CUtensorMap tmap_w1,
                  const __grid_constant__ CUtensorMap tmap_a0, const __grid_constant__ CUtensorMap tmap_a1,
                  const __grid_constant__ StreamParams p) {
    stream_tiles<BN, kSwiglu, kBoth, kSplit>(&tmap_w0, &tmap_w1, &tmap_a0, &tmap_a1, p);
}

// The groups divided between both kinds of tiles (launch_fp8_stream says when), one CTA per SM at a time: the CTAs of `small`
// start as those of `large`, which come first, leave.
template <bool kSwiglu, bool kBoth>
__global__ void __launch_bounds__(kNumThreads, 1)
fp8_divided_kernel(const __grid_constant__ CUtensorMap tmap_w0, const __grid_constant__ CUtensorMap tmap_w1,
                   const __grid_constant__ CUtensorMap tmap_a0, const __grid_constant__ CUtensorMap tmap_a1,
                   const __grid_constant__ CUtensorMap tmap_c0, const __grid_constant__ CUtensorMap tmap_c1, const __grid_constant__ StreamParams large, const __grid_constant__ StreamParams small) {
    if (static_cast<int>(blockIdx.x) < large.ctas) rows_tiles<128, kSwiglu, kBoth>(&tmap_w0, &tmap_w1, &tmap_a0, &tmap_a1, &tmap_c0, &tmap_c1, large);
    else stream_tiles<64, kSwiglu, false, false>(&tmap_w0, &tmap_w1, &tmap_a0, &tmap_a1, small);
}

template <typename... KArgs, typename... Args>
int launch(void (*kern)(KArgs...), int64_t grid, int smem, bool (&configured)[64], cudaStream_t stream, const Args&... args) {
    int dev = 0;
    DSV3_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) {
        set_last_error("fp8_gemm: device ordinal %d is outside the supported range", dev);
        return DSV3_ERR_UNSUPPORTED;
    }
    if (!configured[dev]) {
        DSV3_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        configured[dev] = true;
    }
    DSV3_CUDA_TRY(launch_dependent(kern, dim3(static_cast<unsigned>(grid)), dim3(kNumThreads), smem, stream, args...));
    return DSV3_OK;
}

uint64_t coprime_with(int n) {
    uint64_t mask = ~1ull;
    for (int p : {2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37, 41, 43, 47, 53, 59, 61})
        if (n % p == 0)
            for (int i = p; i < 64; i += p) mask &= ~(1ull << i);
    return mask;
}

// most: no more CTAs than there can be work for
template <int BN, bool kSwiglu, bool kBoth, bool kSplit>
int launch_stream(const CUtensorMap& w0, const CUtensorMap& w1, const CUtensorMap& ta0, const CUtensorMap& ta1, StreamParams prm, int64_t most,
                  int sms, cudaStream_t stream) {
    using C = SCfg<BN, false>;
    static bool configured[64] = {};
    prm.ctas = static_cast<int>(most < sms ? most : sms);
    if (kBoth && !kSplit) prm.coprime = coprime_with(prm.ctas);
    return launch(fp8_stream_kernel<BN, kSwiglu, kBoth, kSplit>, prm.ctas, C::kSmemBytes, configured, stream, w0, w1, ta0, ta1, prm);
}

template <bool kSwiglu, bool kBoth>
int launch_divided(const CUtensorMap& w0, const CUtensorMap& w1, const CUtensorMap& ta0, const CUtensorMap& ta1, const CUtensorMap& c0,
                   const CUtensorMap& c1, StreamParams prm, int64_t most_large, int64_t most_small, int divide, int sms, cudaStream_t stream) {
    constexpr int kLarge = SCfg<128, true>::kSmemBytes, kSmall = SCfg<64, false>::kSmemBytes;
    static bool configured[64] = {};
    StreamParams small = prm;
    prm.min_rows = divide + 1;
    prm.ctas = static_cast<int>(most_large < sms ? most_large : sms);
    if (kBoth) prm.coprime = coprime_with(prm.ctas);
    small.max_rows = divide;
    small.first_cta = prm.ctas;
    small.ctas = divide ? static_cast<int>(most_small < sms ? most_small : sms) : 0;
    return launch(fp8_divided_kernel<kSwiglu, kBoth>, prm.ctas + small.ctas, kLarge > kSmall ? kLarge : kSmall, configured, stream, w0, w1, ta0, ta1,
                  c0, c1, prm, small);
}

}  // namespace

// Token tile for an expected load per group.  Uneven routing puts some groups above the expectation; a group that needs
// a second tile reads its weights a second time (from L2).  Weights on the M side cost only the tokens that are there.  B200, us,
// tile 16 / 32 / 64, one layer: 256 experts of 7168 x 2048 at 2.5 tokens per expert 1253 / 1252 / 1228, 16 1838 / 1813 / 1712, 26
// 2172 / 1912 / 1819; 160 of 5120 x 1536 at 19 733 / 667 / 620, 26 747 / 662 / 649; 64 of 2048 x 1408 at 21 134 / 127 / 129, 31 169 /
// 141 / 143.  Where tiles are cut, narrow ones park and add less: 20 of 160 experts of 5120 x 1536 at 0.3, 0.9 and
// 4.5 tokens 41 / 43 / 45, 52 / 54 / 58, 86 / 88 / 97, 16 of 64 of 2048 x 1408 at 5.6 and 11 46 / 49 / 53, 47 / 50 / 56.  The lines at 4 and 24
// are drawn between the two: with many large experts 64 is ahead below them, with few cut ones 16 above.  Above 40 tokens the groups are divided between two
// kinds: those of more than 64 rows in tiles of 128 with tokens on the M side, which read the weights once for 128 tokens, the
// others in tiles of 64 with the weights there, which multiply no empty rows: an expert layer at these sizes runs at the
// board's power limit, and half of the experts of an unevenly routed layer have fewer than half of the mean.  us, tiles of 64
// for all groups / divided: 256 experts of 7168 x 2048, 25 tokens each 1822 / 1826, 32 1858 / 1873, 38 1898 / 1924, 44 2034 / 1974, 64
// 2456 / 2263; 160 of 5120 x 1536, 34 tokens 699 / 721, 41 722 / 743, 75 962 / 916; 64 of 2048 x 1408, 31 tokens 141 / 144, 38 140 /
// 139, 42 146 / 143, 66 183 / 181.  Tiles of 128 for all groups, 64 tokens of 7168 x 2048: 2555.
constexpr int kDivide = 64;
static_assert(kDivide <= 64, "one tile of stream_tiles<64>");
int stream_tile(int64_t rows_per_group) {
    return rows_per_group <= 4 ? 16 : (rows_per_group <= 24 ? 32 : (rows_per_group <= 40 ? 64 : 128));
}

static size_t tile_workspace_bytes(int bn, int sms);
size_t stream_workspace_bytes(int64_t rows_per_group) { return stream_tile_workspace_bytes(stream_tile(rows_per_group)); }
size_t stream_tile_workspace_bytes(int bn) { return tile_workspace_bytes(bn, num_sms()); }
static size_t tile_workspace_bytes(int bn, int sms) {
    if (bn > 64) return 0;            // of 128 tokens or divided: never cut
    return DSV3_WORKSPACE_HEADER_BYTES + static_cast<size_t>(sms) * 2 * (2 * bn) * kPRows * sizeof(float);
}

static int fill_side(Side& d, CUtensorMap* map, const StreamSide& q, bool swiglu, int bn) {
    const int rc = make_tmap(map, q.a, q.rows, q.K, bn < 32 ? bn : 32);
    if (rc != DSV3_OK) return rc;
    d.kc = static_cast<int>((q.K + kChunk - 1) / kChunk);
    d.nblk = static_cast<int>((q.N + kPRows - 1) / kPRows);
    d.tiles_p = swiglu ? d.nblk : (d.nblk + 1) / 2;
    d.rows = static_cast<int>(q.rows);
    d.a_s = q.a_s;
    d.as_row = q.as_row;
    d.as_chunk = q.as_chunk;
    d.c = static_cast<__nv_bfloat16*>(q.c);
    d.N = q.N;
    d.vec_store = (q.N % 8) == 0 && (reinterpret_cast<uintptr_t>(q.c) % 16) == 0;
    d.hq = static_cast<uint8_t*>(q.hq);
    d.hs = q.hs;
    d.hs_row = q.hs_row;
    d.hs_blk = q.hs_blk;
    return DSV3_OK;
}

// A launch whose arguments have been looked at.
namespace {
struct StreamLaunch {
    StreamParams prm;
    CUtensorMap w0, w1, ta0, ta1, c0, c1;       // c0, c1: results of tiles of 128 tokens
    int bn, sms, divide;
    bool swiglu, ordinary, split;
    int64_t bound, small;                       // tiles at most (cut tiles: K chunks); of groups of one token tile
};
}  // namespace

static int plan_stream(const StreamGemm& q, StreamLaunch& l) {
    memset(&l, 0, sizeof(l));
    StreamParams& prm = l.prm;
    CUtensorMap &w0 = l.w0, &w1 = l.w1, &ta0 = l.ta0, &ta1 = l.ta1;
    int rc;
    const bool ordinary = q.ordinary.rows > 0;
    const int64_t per_tile = q.n_groups > 0 ? (q.rows_expected + q.n_groups - 1) / q.n_groups : q.ordinary.rows;
    const int bn = q.tile ? q.tile : stream_tile(per_tile);
    int64_t tiles[2] = {0, 0};
    if (q.n_groups > 0) {
        if ((rc = fill_side(prm.side[kGroups], &ta0, q.groups, q.swiglu, bn)) != DSV3_OK) return rc;
        for (int b = 0; b < 2; ++b) {
            const void* tbl = (b == 1 && q.swiglu) ? q.table1 : q.table0;
            prm.g_map[b] = static_cast<const CUtensorMap*>(tbl);
            prm.g_scale[b] = table_scales(tbl, q.n_groups);
        }
        prm.seg = q.seg;
    }
    // token tiles: at most one partly filled tile per group on top of the full ones, and never more groups than rows
    if (q.n_groups > 0)
        tiles[0] = (q.groups.rows / bn + (q.n_groups < q.groups.rows ? q.n_groups : q.groups.rows)) * prm.side[kGroups].tiles_p;
    if (ordinary) {
        const StreamSide& d = q.ordinary;
        if ((rc = fill_side(prm.side[kOrdinary], &ta1, d, q.swiglu, bn)) != DSV3_OK) return rc;
        if ((rc = make_tmap(&w0, q.w0, d.N, d.K, kPRows)) != DSV3_OK) return rc;
        if ((rc = make_tmap(&w1, q.swiglu ? q.w1 : q.w0, d.N, d.K, kPRows)) != DSV3_OK) return rc;
        prm.scale[0] = q.w0_s;
        prm.scale[1] = q.swiglu ? q.w1_s : q.w0_s;
        tiles[1] = (d.rows + bn - 1) / bn * prm.side[kOrdinary].tiles_p;
        if (q.n_groups == 0) ta0 = ta1;                       // (a kernel prefetches both)
    }
    prm.n_groups = q.n_groups;
    prm.max_rows = INT32_MAX;
    prm.scale_fmt = q.scale_fmt;
    prm.leads = q.leads ? 1 : 0;
    prm.early = q.early ? 1 : 0;
    prm.status = status_device_ptr();
    if (!prm.status) return DSV3_ERR_CUDA;
    // cutting tiles is worth considering when one or two rounds of whole tiles are expected (struct Plan)
    const int sms = num_sms();                                // once: the grid must fit the workspace, whatever budget is set meanwhile
    const size_t need = tile_workspace_bytes(bn, sms);
    const int64_t groups_expected = q.n_groups < q.rows_expected ? q.n_groups : q.rows_expected;
    const int64_t tiles_expected = q.n_groups > 0 ? groups_expected * prm.side[kGroups].tiles_p : tiles[1];
    const bool split = bn < 128 && tiles_expected < 3 * sms && q.workspace && q.workspace_bytes >= need &&
                       (reinterpret_cast<uintptr_t>(q.workspace) % 256) == 0;
    if (split) {
        prm.tickets = static_cast<int*>(q.workspace);
        prm.partials = reinterpret_cast<float*>(static_cast<uint8_t*>(q.workspace) + DSV3_WORKSPACE_HEADER_BYTES);
    }
    const int64_t units = tiles[0] * prm.side[kGroups].kc + tiles[1] * prm.side[kOrdinary].kc;
    if (units >= (1ll << 31)) {
        set_last_error("fp8 stream GEMM: %lld K chunks are more than the work-item counter holds", static_cast<long long>(units));
        return DSV3_ERR_UNSUPPORTED;
    }
    if (bn == 128 && !q.swiglu)
        for (int i = 0; i < 2; ++i) {
            const Side& d = prm.side[i];
            if (d.c && d.vec_store && (rc = make_tmap_out(i == kGroups ? &l.c0 : &l.c1, d.c, d.rows, d.N, 32)) != DSV3_OK) return rc;
        }
    if (bn != 16 && bn != 32 && bn != 64 && bn != 128) return DSV3_ERR_UNSUPPORTED;
    l.bn = bn;
    l.sms = sms;
    l.divide = sm_budget_set() ? 0 : kDivide;       // under a budget both kinds' CTAs could be resident side by side
    l.swiglu = q.swiglu;
    l.ordinary = ordinary;
    l.split = split;
    l.bound = split ? units : tiles[0] + tiles[1];
    l.small = (q.n_groups < q.groups.rows ? q.n_groups : q.groups.rows) * prm.side[kGroups].tiles_p;    // (a group of at most kDivide rows is one token tile)
    return DSV3_OK;
}

static int launch_planned(const StreamLaunch& l, cudaStream_t stream) {
#define DSV3_STREAM_LAUNCH(BN_, SW_, SPLIT_)                                                                               \
    return l.ordinary ? launch_stream<BN_, SW_, true, SPLIT_>(l.w0, l.w1, l.ta0, l.ta1, l.prm, l.bound, l.sms, stream)          \
                      : launch_stream<BN_, SW_, false, SPLIT_>(l.w0, l.w1, l.ta0, l.ta1, l.prm, l.bound, l.sms, stream)
#define DSV3_STREAM_CASE(BN_)                                                                                              \
    case BN_:                                                                                                              \
        if (l.swiglu) { if (l.split) DSV3_STREAM_LAUNCH(BN_, true, true); DSV3_STREAM_LAUNCH(BN_, true, false); }          \
        if (l.split) DSV3_STREAM_LAUNCH(BN_, false, true);                                                                 \
        DSV3_STREAM_LAUNCH(BN_, false, false)
#define DSV3_DIVIDED_LAUNCH(SW_)                                                                                           \
    return l.ordinary ? launch_divided<SW_, true>(l.w0, l.w1, l.ta0, l.ta1, l.c0, l.c1, l.prm, l.bound, l.small, l.divide, l.sms, stream) \
                      : launch_divided<SW_, false>(l.w0, l.w1, l.ta0, l.ta1, l.c0, l.c1, l.prm, l.bound, l.small, l.divide, l.sms, stream)
    switch (l.bn) {
        DSV3_STREAM_CASE(16);
        DSV3_STREAM_CASE(32);
        DSV3_STREAM_CASE(64);
        default:
            if (l.swiglu) DSV3_DIVIDED_LAUNCH(true);
            DSV3_DIVIDED_LAUNCH(false);
    }
#undef DSV3_STREAM_LAUNCH
#undef DSV3_STREAM_CASE
#undef DSV3_DIVIDED_LAUNCH
}

int launch_fp8_stream(const StreamGemm& q, cudaStream_t stream) {
    StreamLaunch l;
    const int rc = plan_stream(q, l);
    return rc != DSV3_OK ? rc : launch_planned(l, stream);
}

int launch_fp8_streams(const StreamGemm& first, const StreamGemm& second, cudaStream_t stream) {
    StreamLaunch l[2];
    int rc;
    if ((rc = plan_stream(first, l[0])) != DSV3_OK || (rc = plan_stream(second, l[1])) != DSV3_OK) return rc;
    return (rc = launch_planned(l[0], stream)) != DSV3_OK ? rc : launch_planned(l[1], stream);
}

// The table holds, in device memory, n tensor maps, n scale pointers and n weight pointers.
size_t group_table_bytes(int n) { return static_cast<size_t>(n) * (sizeof(CUtensorMap) + sizeof(const float*) + sizeof(const uint8_t*)); }

int build_group_table(void* table_dev, const void* const* weights, const float* const* scales, int n, int64_t N,
                      int64_t K, cudaStream_t stream) {
    if (n <= 0 || n > kMaxGroupsOfTable) {
        set_last_error("group table: between 1 and %d groups are supported (got %d)", kMaxGroupsOfTable, n);
        return DSV3_ERR_UNSUPPORTED;
    }
    if ((K % 16) != 0 || (reinterpret_cast<uintptr_t>(table_dev) % 64) != 0) {
        set_last_error("group table: needs K %% 16 == 0 and a 64-byte aligned table");
        return DSV3_ERR_UNSUPPORTED;
    }
    std::vector<uint8_t> host(group_table_bytes(n));
    CUtensorMap* maps = reinterpret_cast<CUtensorMap*>(host.data());
    const float** sp = reinterpret_cast<const float**>(host.data() + static_cast<size_t>(n) * sizeof(CUtensorMap));
    const void** wp = reinterpret_cast<const void**>(sp + n);
    for (int e = 0; e < n; ++e) {
        if (!weights[e] || !scales[e] || (reinterpret_cast<uintptr_t>(weights[e]) % 16) != 0) {
            set_last_error("group table: weight %d is null or not 16-byte aligned", e);
            return DSV3_ERR_INVALID_ARGUMENT;
        }
        CUtensorMap m;
        const int rc = make_tmap(&m, weights[e], N, K, kPRows);
        if (rc != DSV3_OK) return rc;
        memcpy(maps + e, &m, sizeof(m));
        sp[e] = scales[e];
        wp[e] = weights[e];
    }
    DSV3_CUDA_TRY(cudaMemcpyAsync(table_dev, host.data(), host.size(), cudaMemcpyHostToDevice, stream));
    DSV3_CUDA_TRY(cudaStreamSynchronize(stream));   // `host` goes out of scope
    return DSV3_OK;
}

}  // namespace dsv3
