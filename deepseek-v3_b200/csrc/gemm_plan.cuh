// Internal interface of the tcgen05 fp8_gemm kernels: problem geometry ("plan") and launcher.
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace dsv3 {

// Geometry chosen for a problem; shared by the workspace query and the launch.
struct TcPlan {
    int error;  // DSV3_OK, or the status to return (detail recorded): a pinned kernel / split factor that cannot be honoured
    bool swap;  // true: weights on the MMA M axis (small M)
    bool pair;  // token-major tiles on CTA pairs (fp8_gemm_tm.cu); never with split-K
    bool wide;  // with pair: 256 x 256 tiles (fp8_gemm_tw.cu)
    bool cluster;   // the splits of a tile form a cluster and meet in shared memory
    int bn;     // rows of the second operand tile
    int tiles_p, tiles_q, splits, kc;
};

bool tc_supported(const void* a, const void* b, const void* c, int64_t M, int64_t N, int64_t K);
TcPlan tc_plan(int64_t M, int64_t N, int64_t K, int force_kernel, int force_split);
// 0 when the plan does not split K; otherwise ticket header + splits * M * N fp32 partial sums.
size_t tc_workspace_bytes(const TcPlan& pl, int64_t M, int64_t N);
int launch_fp8_gemm_tc(const void* a, const float* a_s, const void* b, const float* b_s, int64_t M, int64_t N,
                       int64_t K, void* c, void* workspace, size_t workspace_bytes, const TcPlan& pl,
                       cudaStream_t stream);

// Tensor maps over the operands as they lie in memory.  Operand: [rows, K] bytes, row-major; box = 128 bytes x
// box_rows, 128-byte swizzle, zero fill outside.  Result: [M, N] bf16, row-major; box = 64 columns x 128 (or box_rows) rows,
// 128-byte swizzle (N % 8 == 0).
int make_tmap(CUtensorMap* map, const void* base, int64_t rows, int64_t K, int box_rows);
int make_tmap_out(CUtensorMap* map, void* base, int64_t M, int64_t N, int box_rows = 128);

// Token-major kernel on CTA pairs (256 x 128 tiles, tcgen05 cta_group::2, no split-K): fp8_gemm_tm.cu.
bool tm_pair_supported(int64_t M, int64_t N, int64_t K);
int launch_fp8_gemm_tm(const void* a, const float* a_s, const void* b, const float* b_s, int64_t M, int64_t N,
                       int64_t K, void* c, cudaStream_t stream);

// Token-major kernel on CTA pairs with 256-wide accumulators (256 x 256 tiles, no split-K): fp8_gemm_tw.cu.
bool tw_pair_supported(int64_t M, int64_t N, int64_t K);
// Width of the strips that the tiles of a last round of `tiles` are cut into on a machine of `pairs` (0: not cut).
int tw_strip_width(int64_t tiles, int64_t pairs, int kc);
int launch_fp8_gemm_tw(const void* a, const float* a_s, const void* b, const float* b_s, int64_t M, int64_t N,
                       int64_t K, void* c, cudaStream_t stream);
// Two weights of one size on the same activations in one launch: w1 and w3 of an MLP.
int launch_fp8_gemm_tw_two(const void* a, const float* a_s, const void* const (&b)[2], const float* const (&b_s)[2], int64_t M, int64_t N, int64_t K,
                           void* const (&c)[2], cudaStream_t stream);
bool tw_two_pay(int64_t M, int64_t N, int64_t K);

// Decode-sized Linear without tcgen05 set-up (fp8_linear_small.cu): M <= 16; x != nullptr quantises bf16 activations
// in the kernel's prologue (K % 128 == 0), otherwise (a, a_s) are the quantised activations (K % 16 == 0).
bool small_linear_supported(const void* act, const void* w, const void* c, int64_t M, int64_t N, int64_t K, bool fused);
bool decode_kernel_pays(int64_t M, int64_t N, int64_t K);
int launch_fp8_linear_small(const void* x, const void* a, const float* a_s, const void* w, const float* w_s, int64_t M,
                            int64_t N, int64_t K, int scale_fmt, void* c, cudaStream_t stream);

// Weight-streaming GEMM (fp8_stream.cu): groups of rows against per-group weights and, in the same launch, one ordinary
// weight; optionally with SwiGLU of two weights and quantisation of the product in the epilogue.
struct StreamSide {
    const void* a;                     // e4m3 [rows, K]
    const float* a_s;                  // token scales at a_s[row * as_row + chunk * as_chunk]
    int64_t as_row, as_chunk;
    int64_t rows, N, K;
    void* c;                           // bf16 [rows, N]                   -- plain
    void* hq;                          // e4m3 [rows, N]                   -- swiglu
    float* hs;                         // hs[row * hs_row + block * hs_blk] -- swiglu
    int64_t hs_row, hs_blk;
};
struct StreamGemm {
    StreamSide groups;
    int n_groups;
    int64_t rows_expected;             // rows the groups are expected to own together
    const void *table0, *table1;       // group tables; table1 only with swiglu
    const int* seg;                    // device memory
    StreamSide ordinary;               // rows == 0: none
    const void *w0, *w1;               // e4m3 [N, K]; w1 only with swiglu
    const float *w0_s, *w1_s;
    bool swiglu;
    // early: the launch before this one on the stream is another of these, with `leads`, and only its results (a, a_s, and c's memory) have to be waited
    // for: row offsets, tables and weights are read while it still runs.  They are complete by then, since it lets its dependents
    // start only once what came before it has finished.  w2's CTAs plan their tiles and fill their rings with weights on the SMs that
    // w1's and w3's have left; us per layer, without / with: 64 experts of 2048 x 1408, 7 and 333 tokens 61.7 / 57.3, 135.0 / 132.6, 8 of them
    // and 62 39.9 / 37.6; 20 of 160 of 5120 x 1536, 442 145.4 / 138.8, all 160 and 40 356.5 / 353.0; two layers of a decode step, one rank of
    // eight, 16 sequences 230.2 / 223.3; 256 experts of 7168 x 2048, 2048 tokens 2373 / 2379 (their runs differ by 1 %).
    bool leads, early;
    int scale_fmt;
    int tile;                          // tokens per tile (16, 32, 64, 128), or 0: by rows_expected
    void* workspace;                   // stream_workspace_bytes(), or null: tiles are not split
    size_t workspace_bytes;
};
// Whether a last round is cut over K, and into how many ranges (0: tiles are worked on whole).  tiles, units: of the whole problem, a
// unit being one K chunk of a tile; last: units of the last round; longest: chunks of its longest tile.  Time of that round, in
// sixteenths of the 0.75 us a chunk takes with every SM loading: whole tiles are bound by what one CTA folds when it has HBM to
// itself, an even cut by HBM, plus parking and adding up, three chunks (B200: 64 tokens of a decode layer's 32 experts, one round,
// 464 us whole, 410 cut).  A range is at least three 32 KB chunks.
__host__ __device__ inline int cut_ranges(int bn, int tiles, int units, int last, int longest, int ctas) {
    const int alone = bn <= 32 ? 7 : 9;
    if (bn > 64 || longest * alone <= static_cast<int>(16u * static_cast<unsigned>(last) / static_cast<unsigned>(ctas)) + 16 * 3) return 0;
    const int by_size = units / 3 > 1 ? units / 3 : 1, ranges = ctas < by_size ? ctas : by_size;
    return ranges > tiles || ranges == ctas ? ranges : 0;
}
int stream_tile(int64_t rows_per_group);
size_t stream_workspace_bytes(int64_t rows_per_group);
size_t stream_tile_workspace_bytes(int bn);
int launch_fp8_stream(const StreamGemm& q, cudaStream_t stream);
// One after the other; nothing is launched where either is refused.
int launch_fp8_streams(const StreamGemm& first, const StreamGemm& second, cudaStream_t stream);

// Table of the weights of up to 256 groups: tensor maps, scale pointers and weight pointers, in device memory.
constexpr int kMaxGroupsOfTable = 256;
constexpr int kMaxTopk = 32;       // experts per token, whichever form of the expert layer takes the call
size_t group_table_bytes(int n);
inline const float* const* table_scales(const void* table, int n) {
    return reinterpret_cast<const float* const*>(static_cast<const uint8_t*>(table) + static_cast<size_t>(n) * sizeof(CUtensorMap));
}
inline const uint8_t* const* table_weights(const void* table, int n) { return reinterpret_cast<const uint8_t* const*>(table_scales(table, n) + n); }
int build_group_table(void* table_dev, const void* const* weights, const float* const* scales, int n, int64_t N,
                      int64_t K, cudaStream_t stream);

// One thread waits for an mbarrier phase that never completes; the bounded wait gives up after limit_ns.
int launch_bounded_wait_selftest(uint64_t limit_ns, cudaStream_t stream);

// Kernel / split-K override set through dsv3_set_gemm_policy (0 = automatic).
int gemm_policy_kernel();
int gemm_policy_split();

}  // namespace dsv3
