// Batched tree growth ("waves").
//
// The reference grows a tree leaf-wise, one split per iteration: the leaf of largest
// cached gain is split, its smaller child histogrammed, the larger derived by
// subtraction (cpp/src/tree.cpp:343-463).  Done literally on a GPU that is one chain of
// small launches per split.  A wave does the same work for many leaves, and for many
// trees (the folds of a walk-forward split, or any set of fit contexts), per launch:
//
//   select    replays the best-first choice exactly: while the best candidate leaf
//             (largest gain, lowest node id on ties; tree.cpp:343-383) has already been
//             expanded, it is committed: node ids, children, split records, exactly as
//             the one-split loop creates them.  It stops at the first unexpanded best
//             leaf, or when the tree is done, then plans the next expansions: every
//             unexpanded leaf among the top-B candidates, B = the splits left.  No leaf
//             outside the top B can ever be chosen (the B better ones exhaust the
//             budget first), and the best one is always expanded, so every wave commits
//             at least one split and the result is the reference's tree.
//   partition the planned leaves' rows into their children (tree.cpp:68-91), into the
//             other ping-pong buffer at the leaf's own row range: a leaf whose expansion
//             is never committed keeps its rows untouched.  The order of the rows inside a
//             child is free: everything computed from a row list is an exact integer sum.
//   histogram the smaller child of every planned leaf, one persistent cluster launch
//             over all (context, leaf) jobs: rows x feature groups cut into one
//             contiguous range per cluster, or, where there are clusters enough, clusters
//             of its own for every (job, group).
//   scan      both children of every planned leaf (the larger by parent - smaller,
//             histogram.cpp:108-117) for their best split and their totals.
//
// Histogram slots are handed out per expansion (slot 0: the root; expansion k of a tree
// gets slots 1 + 2k and 2 + 2k), so speculative children never overwrite committed
// ones.  A tree has at most 2 * max_leaves - 1 committed nodes and each is expanded at
// most once, so 4 * max_leaves - 1 slots always suffice.
#pragma once

#include <cuda.h>

#include "tgb_internal.h"

namespace tgb {

constexpr int kMaxWaveCtx = 64;     // fit contexts per wave launch
constexpr int kMaxLeavesCap = 256;  // max_leaves limit of the GPU path
constexpr int kMaxWaveJobs = 4096;  // (context, expansion) pairs per histogram launch

// Histogram payload (what one row contributes) and its accumulation:
//   exact: 64-bit fixed point per row, exact integer sums (results match the reference)
//   q16 / q8: gradients (and hessians) stochastically rounded to 16 / 8 bits per tree,
//   summed exactly in 32-bit shared words (the precision pattern)
// const: unit hessians (mse), H is rebuilt from row counts; var: per-row hessians.
enum HistMode : int {
    kHistExactConst = 0,
    kHistExactVar = 1,
    kHistQ16Const = 2,
    kHistQ16Var = 3,
    kHistQ8Const = 4,
    kHistQ8Var = 5,
};
inline int hist_mode(int hist_bits, bool const_h) {
    const int base = hist_bits == 16 ? kHistQ16Const : hist_bits == 8 ? kHistQ8Const : kHistExactConst;
    return base + (const_h ? 0 : 1);
}
// Bytes of a row's histogram payload in `mode` (the g payload; the exact per-row mode adds
// an 8-byte h payload).
inline int hist_pay_bytes(int mode) { return mode <= kHistExactVar ? 8 : mode <= kHistQ16Var ? 4 : 2; }

// What the partition reads of a planned expansion, written whole by the select that plans
// it: the leaf's rows and slot, its children's first slot, and the split.
struct alignas(16) WaveExp {
    int leaf, start, count, buf;
    int feature, threshold, missing_left, type;
    int feature2, depth, slot, child_slot;
    unsigned long long cat[4];
};

// What the histogram and the scan read of a planned expansion, written whole by the
// partition tile that completes the leaf: one load instead of a chain through the node
// table.  WaveJob: the smaller child's rows (cpp/src/tree.cpp:423) and slot.  WaveChild:
// candidate index, slot, and the parent and small-sibling slots the larger child's
// histogram is derived from.
struct alignas(16) WaveJob {
    int start, count, buf, slot;
};
struct alignas(16) WaveChild {
    int ci, slot, pslot, sslot;
    int derive, eligible, pad[2];
};

// Per-tree control of one context, device resident.
struct WaveCtl {
    int splits_done;  // splits committed so far
    int n_exp;        // expansions planned by the last select
    int exp_counter;  // expansions so far in this tree (slot hand-out)
    int tiles_total;  // partition tiles of the planned expansions
    int active;       // 1 while the tree grows
    int slot0;        // first histogram slot of the planned expansions
    // a slot, buffer or wave-count bound was hit, or a staging wait gave up (never expected): the
    // first such code of the fit, zeroed with the fit's buffers and read after its last tree
    int error;
    int waves;        // selects run for this tree (bounded: a tree needs at most max_leaves)
    int pair_used;    // PAIR splits committed in this tree
    int exp_total;    // expansions planned over all trees of the fit (not reset per tree)
    int pad[2];
    int exp_tile0[kMaxLeavesCap + 1];
    // rows of the planned leaf placed so far by its partition tiles: left in the low word,
    // right in the high word (zeroed by the select that plans the expansion)
    unsigned long long part_cur[kMaxLeavesCap];
    WaveExp exp[kMaxLeavesCap];            // per planned expansion
    WaveJob job[kMaxLeavesCap];
    WaveChild child[2 * kMaxLeavesCap];    // per planned expansion and side
    int expanded[kMaxNodes];  // 0 not expanded; 1, 2: children planned by the axis, with-pairs split
};

// Everything a wave kernel needs to know about one context (device resident array).
struct WaveCtx {
    // TMA descriptor of codes (uint8 [n][stride], box: 32 bytes of one row) for the
    // histogram's gathers; used when codes_map_ok (encode_codes_map succeeded)
    CUtensorMap codes_map;
    const uint8_t* codes;      // row-major [n][stride]
    const uint8_t* codes_col;  // column-major [F][col_pitch]
    long long col_pitch;
    int32_t* rows0;
    int32_t* rows1;
    // Histogram payloads by position: the payload of the row at position k of rows buffer b
    // (rows0: b = 0, rows1: b = 1) is element b * pay_pitch + k of gq (pay_bytes bytes) and
    // of hq (8 bytes, exact per-row hessian mode only); the partition moves them with the
    // rows, so the histogram reads them in row-list order.
    void* gq;
    void* hq;
    long long pay_pitch;
    int pay_bytes;
    int pad_pay;
    DevNode* nodes;
    DevSplit* splits;
    DevTreeState* st;
    DevNode* spec;        // [2 * kMaxNodes]: children of node k at 2k, 2k + 1
    DevSplit* spec_split;  // their best splits
    WaveCtl* ctl;
    long long* G;  // histogram slots [n_slots][F][kBins]
    long long* H;
    int* C;
    double* cand_gain;  // scan candidates [(2 * kMaxNodes + 1)][F]
    int* cand_key;
    int* tickets;      // [2 * kMaxNodes + 1], zero between launches
    GrowParams gp;
    double goss_scale;
    int n_slots;
    int max_tiles;
    int max_expand;  // expansions a select may plan (0: every candidate ranked within the budget)
    int codes_map_ok;
    // categorical features (nullptr: none): flags per feature, the left masks of the scan
    // candidates [(2 * kMaxNodes + 1)][F][4], and the ranking's smoothing (cat_smooth)
    const uint8_t* is_cat;
    unsigned long long* cand_cat;
    double cat_smooth;
    // PAIR splits (tree.cpp:214-281; pair_on 0: off).  A leaf whose best axis gain is weak
    // against its gradient energy also tries the pairs of its top-k features through the
    // histogram of the hashed code pair; splits_pair / spec_split_pair hold the best split
    // with those pairs (the split a leaf takes while the tree's pair budget lasts), splits /
    // spec_split the one without.  energy: per candidate index, fixed point (2^-energy_shift
    // of the rows' sum of g^2).
    int pair_on;
    int pair_top_k;
    int max_pair;
    int pad_pair;
    double pair_trigger;
    double pair_l2;
    const double* g;           // the rows' gradients (the tree's g before GOSS scaling)
    const uint8_t* goss_flag;  // GOSS classes (nullptr: no GOSS); class 2 rows are scaled
    DevSplit* splits_pair;
    DevSplit* spec_split_pair;
    unsigned long long* energy;  // [2 * kMaxNodes + 1]
    // pair histograms of the wave's children, [pair_children][kMaxPairs][kBins] each, and the
    // chunks done per candidate index [2 * kMaxNodes + 1]; all zero between launches
    unsigned long long* pair_G;
    unsigned long long* pair_H;
    int* pair_C;
    int* pair_tickets;
};
constexpr int kMaxPairs = 15;  // pairs of the top pair_top_k <= 6 features

#if defined(__CUDACC__)
// The fixed-point shift of the gradient energies: no sum over the sample reaches 2^62.
__device__ __forceinline__ int energy_shift(const DevTreeState* st) {
    const double mg = __longlong_as_double(static_cast<long long>(st->max_abs_g_bits));
    const double e2 = mg * mg;
    const int n = st->n_sample;
    if (!(e2 > 0.0) || n <= 0) return 0;
    const int clog = n > 1 ? 32 - __clz(n - 1) : 0;
    return max(-1000, min(1000, 61 - (ilogb(e2) + 1) - clog));
}

// Notes an error of the fit; a later one does not replace it.
__device__ __forceinline__ void set_error(int* error, int code) { atomicCAS(error, 0, code); }

// Copies the first context into shared memory (the caller synchronises the CTA).  The
// contexts are written before the fit's first tree and do not change, so a wave kernel does
// this before pdl_wait: its later reads of pointers and parameters then cost no memory
// round trip of their own.
__device__ __forceinline__ void stage_ctx(WaveCtx& to, const WaveCtx* ctxs) {
    static_assert(sizeof(WaveCtx) % 16 == 0, "copied in 16-byte words");
    const uint4* src = reinterpret_cast<const uint4*>(ctxs);
    uint4* dst = reinterpret_cast<uint4*>(&to);
    for (int k = threadIdx.x; k < static_cast<int>(sizeof(WaveCtx) / 16); k += blockDim.x) dst[k] = __ldg(src + k);
}
#endif

// Children a wave may hold (two per planned expansion; at least the root).
inline int wave_children(int max_leaves, int max_expand) {
    const int e = max_leaves - 1;
    return 2 * (max_expand > 0 && max_expand < e ? max_expand : e);
}

// Per-tree set-up of one context: all-row scales, root node, control reset, histogram scales; the
// root's slot (slot 0 of G, H, C), seg_sums and energy (may be null) cleared; rows0 = 0 .. n - 1
// unless `sampled` (GOSS: the sample is in rows0 and st->n_sample).
struct WaveBegin {
    DevNode* nodes;
    DevSplit* splits;
    DevTreeState* st;
    WaveCtl* ctl;
    AllScale* all;
    long long* G;
    long long* H;
    int* C;
    size_t slot_elems;
    unsigned long long* seg_sums;
    size_t seg_words;
    unsigned long long* energy;
    int32_t* rows0;
    int n, sampled, mode;
};
void launch_wave_begin(const WaveBegin& a, cudaStream_t s);
// Per-tree histogram scales of one context from the sample maxima (st) or, when the
// sample is every row, the all-row maxima (all).
void launch_wave_scales(DevTreeState* st, const AllScale* all, int mode, cudaStream_t s);
// Payload of the sampled rows for `mode` (rows0[0 .. st->n_sample)), by position in rows0.
// The stochastic rounding's stream is `seed`, or with per_tree SplitMix64 of seed + st->tree.
// energy (PAIR, else nullptr; zeroed by the caller): the root's gradient energy.
void launch_wave_quantize(int mode, const int32_t* rows, const double* g, const double* h, const uint8_t* goss_flag,
                          double goss_scale, const DevTreeState* st, unsigned long long seed, bool per_tree, void* gq,
                          void* hq, unsigned long long* energy, int max_rows, cudaStream_t s);

// Wave launches over n_ctx contexts (ctxs: device array).  src 0: the roots, src 1: the
// expansions planned by the last select.
// Launch shape of the histogram: `cluster` CTAs per cluster (1, 2 or 4: how many private
// histograms one flush merges through distributed shared memory), `clusters` clusters
// (co-resident).  Picked by the autotuner.
struct HistTune {
    int cluster = 4;
    int clusters = 37;
};
int wave_hist_clusters(int cluster);  // co-resident clusters of the histogram kernel
// codes_map for a row-major uint8 code matrix [n_rows][stride]: false (map zeroed) where
// TMA cannot address it (stride not a multiple of 16 or below 32 bytes, base not 16-byte
// aligned, no driver entry point); the histogram then loads code rows directly.
bool encode_codes_map(CUtensorMap* map, const uint8_t* codes, long long n_rows, int stride);
void launch_wave_hist(int mode, const WaveCtx* ctxs, int n_ctx, int src, HistTune tune,
                      unsigned long long* rows_counter, cudaStream_t s);
void launch_wave_scan(const WaveCtx* ctxs, int n_ctx, int src, int max_f, int ys, bool any_cat, cudaStream_t s);
// gsync: 3 device ints (flag, ticket, selects run so far), zeroed before the first select.
// host_flag: mapped host word or nullptr; cond / use_cond: the condition of a node of the graph,
// set to "any context still growing".
void launch_wave_select(const WaveCtx* ctxs, int n_ctx, int* gsync, unsigned* host_flag,
                        unsigned long long cond, int use_cond, cudaStream_t s);
void launch_wave_partition(const WaveCtx* ctxs, int n_ctx, int grid, bool pair, cudaStream_t s);
// PAIR stage after a scan (contexts with pair_on): for the children (or roots) whose best
// axis gain is weak against their gradient energy the pair histograms and their best
// splits, merged into spec_split_pair (roots: splits_pair[0]).  var: per-row hessians.
void launch_wave_pair(const WaveCtx* ctxs, int n_ctx, int src, bool var, cudaStream_t s);
void prepare_wave_pair();  // its shared-memory opt-in, once per device (not inside a capture)
// sc->maxg_bits / maxh_bits <- max |g[rows]| and max h[rows] (h == nullptr: 1); sc zeroed.
void launch_rows_max(const int32_t* rows, int n_rows, const double* g, const double* h, AllScale* sc,
                     cudaStream_t s);

}  // namespace tgb
