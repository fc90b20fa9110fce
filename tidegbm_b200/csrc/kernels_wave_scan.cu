// Wave scan and select (wave.h describes the scheme).  Compiled with -fmad=false: the
// gain arithmetic follows the reference's statement order (scan_common.cuh).
//
// scan: one warp per (child, numeric feature), grid-stride over the children of all planned
// leaves of all contexts (or over the roots), one CTA of 256 threads (thread = bin) per
// categorical feature.  The larger child's histogram is derived as parent - smaller child on
// the way (subtract_hist_inplace, cpp/src/histogram.cpp:108-117, exact in fixed point).  The
// last feature of a child to finish (ticket counter, nothing waits) reduces the per-feature
// candidates, lowest feature on ties (best_for_leaf, cpp/src/tree.cpp:120-166).
//
// select: one warp per context.  It commits expanded best leaves in the reference's
// best-first order (grow_tree, cpp/src/tree.cpp:343-383) and plans the next wave's
// expansions; the last context to finish sets the condition of the tree graph's next
// conditional node.
#include "scan_common.cuh"
#include "wave.h"

namespace tgb {

namespace {

using namespace scan;

constexpr int kRootCand = 2 * kMaxNodes;  // candidate / ticket index of the root
constexpr int kMaxPairFeatures = 1024;    // features the PAIR ranking sorts (host-checked)

__device__ __forceinline__ void children_prefix(const WaveCtx* ctxs, int n_ctx, int src, int* s_pref) {
    if (static_cast<int>(threadIdx.x) < n_ctx) {
        const WaveCtl* ctl = ctxs[threadIdx.x].ctl;
        s_pref[threadIdx.x] = src == 0 ? (ctl->active ? 1 : 0) : 2 * ctl->n_exp;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int acc = 0;
        for (int c = 0; c < n_ctx; ++c) {
            const int v = s_pref[c];
            s_pref[c] = acc;
            acc += v;
        }
        s_pref[n_ctx] = acc;
    }
    __syncthreads();
}

// The histogram job of one child (child k of the context's wave, or the root): its
// candidate index, its slot, and (the larger child) the parent and small-sibling slots it is
// derived from.
__device__ __forceinline__ WaveChild scan_child(const WaveCtx& X, int src, int k) {
    if (src != 0) return X.ctl->child[k];
    return WaveChild{kRootCand, 0, 0, 0, 0, 0 < X.gp.max_depth && X.st->n_sample >= 2 * X.gp.min_samples_leaf, {0, 0}};
}
__device__ __forceinline__ DevNode* child_node(const WaveCtx& X, int src, int ci) {
    return src == 0 ? X.nodes : X.spec + ci;
}
__device__ __forceinline__ DevSplit* child_split(const WaveCtx& X, int src, int ci) {
    return src == 0 ? X.splits : X.spec_split + ci;
}

// The last feature job of a child (one warp): the best candidate over its features
// (best_for_leaf's ascending-feature strict '>', tree.cpp:160-166), written as its split.
__device__ __forceinline__ void finish_child(const WaveCtx& X, int ci, DevSplit* out, int lane) {
    const GrowParams& p = X.gp;
    __threadfence();
    Cand b{-1e300, 0x7fffffff};
    for (int k = lane; k < p.n_features; k += 32) {
        const size_t cs = static_cast<size_t>(ci) * p.n_features + k;
        const Cand cd{static_cast<volatile double*>(X.cand_gain)[cs], static_cast<volatile int*>(X.cand_key)[cs]};
        if (better(cd, b)) b = cd;
    }
    b = warp_best(b);
    if (lane == 0) {
        DevSplit sp{};
        sp.gain = b.gain;
        sp.valid = (b.key != 0x7fffffff) && b.gain >= p.min_split_gain;
        sp.feature = sp.valid ? b.key / 512 : -1;
        sp.threshold = sp.valid ? (b.key % 512) / 2 : -1;
        sp.missing_left = sp.valid ? (b.key & 1) : 1;
        sp.type = 0;
        if (sp.valid && X.is_cat != nullptr && X.is_cat[sp.feature]) {
            // categorical: the winning feature's left mask; missing follows bin 0's side
            const unsigned long long* m = X.cand_cat + (static_cast<size_t>(ci) * p.n_features + sp.feature) * 4;
            sp.type = 2;
            sp.threshold = -1;
            for (int k = 0; k < 4; ++k) sp.cat[k] = reinterpret_cast<const volatile unsigned long long*>(m)[k];
            sp.missing_left = static_cast<int>(sp.cat[0] & 1ull);
        }
        *out = sp;
        X.tickets[ci] = 0;  // ready for the next launch
    }
}

// Node totals from feature 0 (every feature's bins sum to the same integers) and the
// node's value (leaf_value, cpp/include/tidegbm/tree.hpp:53-67).
__device__ __forceinline__ void set_totals(DevNode* N, long long Gt, long long Ht, long long Ct, double inv_gs,
                                           double inv_hs, double l2) {
    N->G = Gt;
    N->H = Ht;
    N->C = Ct;
    const double dg = static_cast<double>(Gt) * inv_gs, dh = static_cast<double>(Ht) * inv_hs;
    N->value = -dg / (dh + l2);
}

// Numeric features, one warp per (child, feature): every child's histogram scanned by
// scan_feature_warp (the larger child first derived as parent - smaller), the per-feature
// bests kept as candidates, and the child's last job picks its split.  Categorical
// features are left to wave_scan_cat_kernel; the children's tickets count both.
constexpr int kScanWarpThreads = 128;
constexpr int kScanWarpCtas = 4;  // per SM

__global__ void __launch_bounds__(kScanWarpThreads, kScanWarpCtas)
    wave_scan_warp_kernel(const WaveCtx* __restrict__ ctxs, int n_ctx, int src) {
    __shared__ WaveCtx s_ctx;  // the first context's constants
    __shared__ int s_jpref[kMaxWaveCtx + 1];
    stage_ctx(s_ctx, ctxs);
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    auto ctx_of = [&](int c) -> const WaveCtx& { return c == 0 ? s_ctx : ctxs[c]; };
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < 32) {
        int all = 0;
        for (int c0 = 0; c0 < n_ctx; c0 += 32) {
            const int c = c0 + lane;
            int v = 0;
            if (c < n_ctx) {
                const WaveCtl* ctl = ctx_of(c).ctl;
                v = (src == 0 ? (ctl->active ? 1 : 0) : 2 * ctl->n_exp) * ctx_of(c).gp.n_features;
            }
            int incl = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            if (c < n_ctx) s_jpref[c] = all + incl - v;
            all += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) s_jpref[n_ctx] = all;
    }
    __syncthreads();
    const int wpb = kScanWarpThreads / 32;
    const int total = s_jpref[n_ctx];
    for (int jw = blockIdx.x * wpb + (threadIdx.x >> 5); jw < total; jw += gridDim.x * wpb) {
        int c = 0;
        while (c + 1 < n_ctx && s_jpref[c + 1] <= jw) ++c;
        const WaveCtx& X = ctx_of(c);
        const GrowParams& p = X.gp;
        const int rem = jw - s_jpref[c];
        const int k = rem / p.n_features, f = rem - k * p.n_features;
        if (X.is_cat != nullptr && X.is_cat[f]) continue;
        const WaveChild t = scan_child(X, src, k);
        const size_t e = static_cast<size_t>(p.n_features) * kBins;
        const double inv_gs = X.st->inv_gscale, inv_hs = X.st->inv_hscale;
        Cand best{-1e300, 0x7fffffff};
        if (t.eligible || f == 0) {
            const size_t fo = static_cast<size_t>(f) * kBins;
            const size_t so = static_cast<size_t>(t.slot) * e + fo, po = static_cast<size_t>(t.pslot) * e + fo,
                         qo = static_cast<size_t>(t.sslot) * e + fo;
            long long Gt, Ht, Ct;
            best = scan_feature_warp(X.G + so, X.H + so, X.C + so, X.G + po, X.H + po, X.C + po, X.G + qo, X.H + qo,
                                     X.C + qo, t.derive, t.eligible, f, p.n_bins, inv_gs, inv_hs, p.l2, p.min_split_gain,
                                     p.min_samples_leaf, p.min_child_weight, Gt, Ht, Ct);
            if (f == 0 && lane == 0) set_totals(child_node(X, src, t.ci), Gt, Ht, Ct, inv_gs, inv_hs, p.l2);
        }
        int last = 0;
        if (lane == 0) {
            const size_t cs = static_cast<size_t>(t.ci) * p.n_features + f;
            X.cand_gain[cs] = best.gain;
            X.cand_key[cs] = best.key;
            __threadfence();
            last = atomicAdd(&X.tickets[t.ci], 1) == p.n_features - 1;
        }
        last = __shfl_sync(0xffffffffu, last, 0);
        if (last) finish_child(X, t.ci, child_split(X, src, t.ci), lane);
    }
}

// Categorical features, one CTA per (child, feature): the histogram (derived as above)
// ranked and scanned by scan_categorical (best_categorical, histogram.cpp:195-244).
__global__ void __launch_bounds__(kScanThreads)
    wave_scan_cat_kernel(const WaveCtx* __restrict__ ctxs, int n_ctx, int src) {
    pdl_wait();
    pdl_trigger();
    __shared__ int s_pref[kMaxWaveCtx + 1];
    __shared__ ScanShared sm;
    __shared__ CatShared csm;
    __shared__ int last;
    children_prefix(ctxs, n_ctx, src, s_pref);
    const int total = s_pref[n_ctx];
    const int f = blockIdx.x;
    for (int j = blockIdx.y; j < total; j += gridDim.y) {
        int c = 0;
        while (c + 1 < n_ctx && s_pref[c + 1] <= j) ++c;
        const WaveCtx& X = ctxs[c];
        const GrowParams& p = X.gp;
        if (f >= p.n_features || X.is_cat == nullptr || !X.is_cat[f]) continue;  // uniform over the CTA
        const WaveChild t = scan_child(X, src, j - s_pref[c]);
        const size_t e = static_cast<size_t>(p.n_features) * kBins;
        const bool eligible = t.eligible != 0;
        const double inv_gs = X.st->inv_gscale, inv_hs = X.st->inv_hscale;
        Cand best{-1e300, 0x7fffffff};
        if (eligible || f == 0) {
            const size_t fo = static_cast<size_t>(f) * kBins;
            const size_t so = static_cast<size_t>(t.slot) * e + fo, po = static_cast<size_t>(t.pslot) * e + fo,
                         qo = static_cast<size_t>(t.sslot) * e + fo;
            long long Gt, Ht, Ct;
            best = scan_feature(X.G + so, X.H + so, X.C + so, X.G + po, X.H + po, X.C + po, X.G + qo, X.H + qo,
                                X.C + qo, t.derive, false, f, p.n_bins, inv_gs, inv_hs, p.l2, p.min_split_gain,
                                p.min_samples_leaf, p.min_child_weight, sm, Gt, Ht, Ct);
            if (eligible) {
                // best_categorical over the stored (possibly just derived) histogram
                __syncthreads();
                best = scan_categorical(X.G + so, X.H + so, X.C + so, f, inv_gs, inv_hs, p.l2, p.min_split_gain,
                                        p.min_samples_leaf, p.min_child_weight, X.cat_smooth, Gt, Ht, Ct, csm,
                                        X.cand_cat + (static_cast<size_t>(t.ci) * p.n_features + f) * 4);
            }
            if (f == 0 && threadIdx.x == 0) set_totals(child_node(X, src, t.ci), Gt, Ht, Ct, inv_gs, inv_hs, p.l2);
        }
        if (threadIdx.x == 0) {
            const size_t cs = static_cast<size_t>(t.ci) * p.n_features + f;
            X.cand_gain[cs] = best.gain;
            X.cand_key[cs] = best.key;
            __threadfence();
            last = atomicAdd(&X.tickets[t.ci], 1) == p.n_features - 1;
        }
        __syncthreads();
        if (last && threadIdx.x < 32)
            finish_child(X, t.ci, child_split(X, src, t.ci), static_cast<int>(threadIdx.x));
        __syncthreads();  // shared state reuse
    }
}

// A leaf the reference's selection may pick: depth and size limits, a valid split of gain
// above min_split_gain (tree.cpp:343-383; the strict '>' against min_split_gain).
__device__ __forceinline__ bool candidate(const GrowParams& p, const DevNode& N, const DevSplit& S) {
    // no short circuit: the loads go out together
    return (N.is_leaf != 0) & (N.depth < p.max_depth) & (N.count >= 2 * p.min_samples_leaf) & (S.valid != 0) &
           (S.gain > p.min_split_gain);
}

// A gain as an unsigned integer of the same order (both zeros alike); never 0 for a number.
__device__ __forceinline__ unsigned long long ordered(double g) {
    const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(g + 0.0));
    return (b >> 63) ? ~b : b | 0x8000000000000000ull;
}

constexpr int kSelectThreads = 256;  // all stage the selection state; warp 0 then selects

__global__ void __launch_bounds__(kSelectThreads)
    wave_select_kernel(const WaveCtx* __restrict__ ctxs, int n_ctx, int* gsync, unsigned* host_flag,
                       cudaGraphConditionalHandle cond, int use_cond) {
    __shared__ WaveCtx X;  // this context's constants
    stage_ctx(X, ctxs + blockIdx.x);
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    const GrowParams& p = X.gp;
    WaveCtl* ctl = X.ctl;
    DevTreeState* st = X.st;
    DevNode* nodes = X.nodes;
    DevSplit* splits = X.splits;
    const int lane = threadIdx.x & 31;
    __shared__ unsigned long long s_gain[kMaxLeavesCap + 1];
    __shared__ int s_id[kMaxLeavesCap + 1];
    // Selection state staged once, so that the commit loop reads no global memory: per
    // node its current split's gain, candidacy, type and with-pairs type, and whether it
    // is expanded; per expanded node the same for its two planned children.  Restaged
    // from the node table when the pair budget runs out (the splits change).
    __shared__ unsigned long long s_key[kMaxNodes];  // ordered gain of a candidate, else 0
    __shared__ unsigned char s_ex[kMaxNodes], s_ty[kMaxNodes], s_pty[kMaxNodes];
    __shared__ unsigned long long s_ckey[2 * kMaxNodes];
    __shared__ unsigned char s_cty[2 * kMaxNodes], s_cpty[2 * kMaxNodes];
    __shared__ int s_commit[kMaxLeavesCap];
    int active = 0;
    if (ctl->active) {
        const int budget = p.max_leaves - 1;
        // every select commits at least one split or ends the tree, so a tree takes at most
        // max_leaves of them; past that bound the tree is ended with the error flag set
        const bool runaway = ctl->waves > p.max_leaves + 1;
        int nn = st->n_nodes;
        int done_splits = ctl->splits_done;
        int pair_used = ctl->pair_used;
        // the split a leaf takes: with the PAIR candidates while the tree's pair budget lasts
        // (tree.cpp:214-218, re-scored after every pair split, tree.cpp:393-396)
        auto pairs_on = [&]() { return X.pair_on && pair_used < X.max_pair; };
        // every load of a node before the first use, whether or not it is expanded
        auto stage_all = [&](int t, int step) {
            const bool pr = pairs_on();
            for (int k = t; k < nn; k += step) {
                const DevSplit* Sp = (pr ? X.splits_pair : splits) + k;
                const DevSplit* Cp = (pr ? X.spec_split_pair : X.spec_split) + 2 * k;
                const DevNode &N = nodes[k], &A = X.spec[2 * k], &B = X.spec[2 * k + 1];
                const double g = Sp->gain, g0 = Cp[0].gain, g1 = Cp[1].gain;
                const int ty = Sp->type, ty0 = Cp[0].type, ty1 = Cp[1].type, ex = ctl->expanded[k];
                const bool c = candidate(p, N, *Sp), c0 = candidate(p, A, Cp[0]), c1 = candidate(p, B, Cp[1]);
                s_key[k] = c ? ordered(g) : 0ull;
                s_ty[k] = static_cast<unsigned char>(ty);
                s_ex[k] = static_cast<unsigned char>(ex);
                s_ckey[2 * k] = c0 ? ordered(g0) : 0ull;
                s_ckey[2 * k + 1] = c1 ? ordered(g1) : 0ull;
                s_cty[2 * k] = static_cast<unsigned char>(ty0);
                s_cty[2 * k + 1] = static_cast<unsigned char>(ty1);
                s_pty[k] = X.pair_on ? static_cast<unsigned char>(X.splits_pair[k].type) : 0;
                s_cpty[2 * k] = X.pair_on ? static_cast<unsigned char>(X.spec_split_pair[2 * k].type) : 0;
                s_cpty[2 * k + 1] = X.pair_on ? static_cast<unsigned char>(X.spec_split_pair[2 * k + 1].type) : 0;
            }
        };
        // the node-table writes of the pending commits (children ids nn_first + 2i, + 1 for
        // the i-th), issued in parallel; `pr`: the pair state they were committed under
        int n_commit = 0, nn_first = nn;
        auto flush = [&](bool pr) {
            for (int i = lane; i < n_commit; i += 32) {
                const int bi = s_commit[i], nc = nn_first + 2 * i;
                const DevSplit S = pr ? X.splits_pair[bi] : splits[bi];
                DevNode& P = nodes[bi];
                P.is_leaf = 0;
                P.feature = S.feature;
                P.threshold = S.threshold;
                P.missing_left = S.missing_left;
                P.gain = S.gain;
                P.type = S.type;
                P.feature2 = S.type == 1 ? S.feature2 : -1;
                for (int k = 0; k < 4; ++k) P.cat[k] = S.cat[k];
                P.left = nc;
                P.right = nc + 1;
                nodes[nc] = X.spec[2 * bi];
                nodes[nc + 1] = X.spec[2 * bi + 1];
                splits[nc] = X.spec_split[2 * bi];
                splits[nc + 1] = X.spec_split[2 * bi + 1];
                if (X.pair_on) {
                    X.splits_pair[nc] = X.spec_split_pair[2 * bi];
                    X.splits_pair[nc + 1] = X.spec_split_pair[2 * bi + 1];
                }
                ctl->expanded[nc] = 0;
                ctl->expanded[nc + 1] = 0;
            }
            __syncwarp();
            __threadfence_block();
            n_commit = 0;
            nn_first = nn;
        };
        stage_all(static_cast<int>(threadIdx.x), static_cast<int>(blockDim.x));
        __syncthreads();
        if (threadIdx.x >= 32) return;  // warp 0 selects
        if (lane == 0) ctl->waves += 1;
        bool finished = false;
        while (true) {
            if (done_splits >= budget || runaway) {
                finished = true;
                break;
            }
            // the best candidate: the largest ordered gain (two 32-bit warp maxima), lowest id
            unsigned long long bk = 0ull;
            int bi = 0x7fffffff;
            for (int k = lane; k < nn; k += 32) {
                const unsigned long long key = s_key[k];
                if (key > bk) {
                    bk = key;
                    bi = k;
                }
            }
            const unsigned hi = static_cast<unsigned>(bk >> 32);
            const unsigned top = __reduce_max_sync(0xffffffffu, hi);
            const unsigned lo = hi == top ? static_cast<unsigned>(bk) : 0u;
            const unsigned topl = __reduce_max_sync(0xffffffffu, lo);
            bi = static_cast<int>(
                __reduce_min_sync(0xffffffffu, hi == top && lo == topl ? static_cast<unsigned>(bi) : 0x7fffffffu));
            if (bi == 0x7fffffff) {
                finished = true;
                break;
            }
            const int ex = s_ex[bi];
            if (!ex) break;
            // an expansion planned with bi's PAIR split while the budget lasted is void once the
            // budget is spent (bi now takes its axis split): plan bi again
            if (ex == 2 && !pairs_on() && s_pty[bi] == 1) {
                if (lane == 0) {
                    ctl->expanded[bi] = 0;
                    s_ex[bi] = 0;
                }
                __syncwarp();
                __threadfence_block();
                break;
            }
            // commit: the split of bi, children ids nn, nn + 1 (grow_tree's numbering)
            const bool pr_before = pairs_on();
            const int ty = s_ty[bi];
            if (lane == 0) {
                s_commit[n_commit] = bi;
                s_key[bi] = 0ull;
            }
            if (lane < 2) {
                const int k = nn + lane, ci = 2 * bi + lane;
                s_key[k] = s_ckey[ci];
                s_ex[k] = 0;
                s_ty[k] = s_cty[ci];
                s_pty[k] = s_cpty[ci];
            }
            __syncwarp();
            n_commit += 1;
            nn += 2;
            done_splits += 1;
            if (ty == 1) pair_used += 1;
            if (pr_before != pairs_on()) {
                // the budget ran out: write the commits so far, then axis splits from here
                flush(pr_before);
                stage_all(lane, 32);
                __syncwarp();
            }
        }
        flush(pairs_on());
        int n_exp = 0;
        if (!finished) {
            // candidates of the new state, best first
            int nc = 0;
            for (int k0 = 0; k0 < nn; k0 += 32) {
                const int k = k0 + lane;
                const unsigned long long gk = k < nn ? s_key[k] : 0ull;
                const bool is_c = gk != 0ull;
                const unsigned m = __ballot_sync(0xffffffffu, is_c);
                if (is_c) {
                    const int pos = nc + __popc(m & ((1u << lane) - 1u));
                    if (pos < kMaxLeavesCap) {
                        s_gain[pos] = gk;
                        s_id[pos] = k;
                    }
                }
                nc += __popc(m);
            }
            nc = min(nc, kMaxLeavesCap);
            __syncwarp();
            const int B = budget - done_splits;
            // expansions: unexpanded candidates ranked below B; in candidate (node id) order
            int base_tiles = 0;
            const int slot_first = 1 + 2 * ctl->exp_counter;
            for (int i0 = 0; i0 < nc; i0 += 32) {
                const int i = i0 + lane;
                bool take = false;
                if (i < nc) {
                    // ids ascend with the position, so a tie ranks the earlier one first
                    int rank = 0;
                    const unsigned long long mine = s_gain[i];
#pragma unroll 8
                    for (int q = 0; q < nc; ++q) rank += (s_gain[q] > mine) | ((s_gain[q] == mine) & (q < i));
                    take = rank < B && (X.max_expand <= 0 || rank < X.max_expand) && !s_ex[s_id[i]];
                }
                const unsigned m = __ballot_sync(0xffffffffu, take);
                int tiles = 0;
                int e = n_exp + __popc(m & ((1u << lane) - 1u));
                if (take) {
                    const int L = s_id[i];
                    const DevNode& N = nodes[L];
                    // 2: the children are partitioned by L's with-pairs split, 1: by its axis split
                    const bool pr = X.pair_on && pair_used < X.max_pair;
                    const DevSplit S = pr ? X.splits_pair[L] : splits[L];
                    tiles = (N.count + kPartTile - 1) / kPartTile;
                    ctl->part_cur[e] = 0ull;
                    ctl->expanded[L] = pr ? 2 : 1;
                    ctl->exp[e] = WaveExp{L, N.start, N.count, N.buf, S.feature, S.threshold, S.missing_left, S.type,
                                          S.feature2, N.depth, N.slot, slot_first + 2 * e,
                                          {S.cat[0], S.cat[1], S.cat[2], S.cat[3]}};
                    for (int sd = 0; sd < 2; ++sd) {
                        DevNode ch{};
                        ch.start = N.start;
                        ch.count = 0;
                        ch.buf = 1 - N.buf;
                        ch.depth = N.depth + 1;
                        ch.is_leaf = 1;
                        ch.feature = -1;
                        ch.threshold = -1;
                        ch.missing_left = 1;
                        ch.left = ch.right = -1;
                        ch.parent = L;
                        ch.slot = slot_first + 2 * e + sd;
                        ch.feature2 = -1;
                        X.spec[2 * L + sd] = ch;
                        if (X.pair_on) X.energy[2 * L + sd] = 0ull;
                    }
                }
                // tile prefix in expansion order
                int incl = tiles;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += t;
                }
                if (take) ctl->exp_tile0[e] = base_tiles + incl - tiles;
                base_tiles += __shfl_sync(0xffffffffu, incl, 31);
                n_exp += __popc(m);
            }
            if (lane == 0) {
                ctl->exp_tile0[n_exp] = base_tiles;
                ctl->tiles_total = base_tiles;
                ctl->slot0 = slot_first;
                ctl->exp_counter += n_exp;
                ctl->exp_total += n_exp;
                if (slot_first + 2 * n_exp > X.n_slots || base_tiles > X.max_tiles) set_error(&ctl->error, 1);
            }
            active = n_exp > 0 && slot_first + 2 * n_exp <= X.n_slots && base_tiles <= X.max_tiles;
        }
        if (lane == 0) {
            if (runaway) set_error(&ctl->error, 1);
            st->n_nodes = nn;
            ctl->splits_done = done_splits;
            ctl->pair_used = pair_used;
            ctl->n_exp = active ? n_exp : 0;
            if (!active) {
                ctl->tiles_total = 0;
                ctl->active = 0;
                st->done = 1;
            }
        }
    }
    // the condition: any context still growing (the last context to finish sets it)
    if (threadIdx.x == 0) {
        unsigned v = active ? 1u : 0u;
        bool last = true;
        if (n_ctx > 1) {
            if (active) atomicOr(&gsync[0], 1);
            __threadfence();
            last = atomicAdd(&gsync[1], 1) == n_ctx - 1;
            if (last) {
                __threadfence();
                v = static_cast<unsigned>(atomicExch(&gsync[0], 0));
                gsync[1] = 0;
            }
        }
        if (last) {
            gsync[2] += 1;  // selects run (for the count of launched kernels)
            if (host_flag != nullptr) {
                *reinterpret_cast<volatile unsigned*>(host_flag) = v;
                __threadfence_system();
            }
            if (use_cond) cudaGraphSetConditional(cond, v);
        }
    }
}

// ---- PAIR stage (tree.cpp:214-281) --------------------------------------------------------
//
// A child whose best axis gain is weak against its gradient energy (the rows' sum of g^2, an
// exact fixed-point sum that the partition makes while it moves the rows) also tries the
// pairs of its top features: the histogram of pair_bin(code1, code2) over its rows (exact
// fixed-point sums of the values the main histogram adds), scanned as one numeric feature
// with pair_l2, merged with the axis split (strict '>' in pair order).
//
// The rows of all weak children are cut into chunks of at most kPairChunk rows, spread over
// the grid.  A CTA adds its chunk's rows into every pair's histogram at once: a row's six
// codes and its payload are read once for 15 pairs, and each pair costs three (per-row
// hessians: five) 32-bit shared reductions with the 19-bit split of the main histogram.
// Chunks are added up in global memory; the child's last chunk to finish scans the pairs, a
// warp each, merges them and clears the sums.  Before, one CTA per (child, pair) walked all
// of the child's rows with 64-bit shared atomics (compare-and-swap loops), after a kernel of
// its own for the energies: 66 us of a 141 us wave at 100k x 32 rows.  The 80-tree fit there
// went from 120.9 to 70.5 ms.
constexpr int kPairThreads = 256;
constexpr int kPairWarps = kPairThreads / 32;
constexpr int kPairChunk = 8192;   // the 19-bit low sums stay below 2^32, the counts in 16 bits
constexpr int kPairMinChunk = 512;  // 256 / 512 / 2,048: 100k x 32 60.1 / 60.3 / 62.2 ms, 20k x 32 40.7 / 40.9 / 41.7
constexpr int kPairLo = 19;
constexpr int kPairTop = 6;        // pair_top_k (host-checked)

// The k features of largest gain in the order std::sort leaves them (tree.cpp:223-225).  When
// each of the k largest gains is unlike all others any sort agrees; otherwise (ties, NaN)
// libstdc++'s own order is replayed.  One warp; gains in shared memory.
__device__ __forceinline__ void top_features(const double* gains, int n_f, int k, short* scratch, int* top) {
    const int lane = threadIdx.x & 31;
    bool plain = true;
    for (int f = lane; f < n_f; f += 32) plain &= gains[f] == gains[f];
    int chosen[kPairTop];
#pragma unroll
    for (int r = 0; r < kPairTop; ++r) chosen[r] = -1;
#pragma unroll
    for (int r = 0; r < kPairTop; ++r) {
        if (r >= k) break;
        unsigned long long bk = 0ull;
        int bi = 0x7fffffff;
        bool twice = false;  // the lane's largest gain occurs twice
        for (int f = lane; f < n_f; f += 32) {
            bool used = false;
#pragma unroll
            for (int q = 0; q < r; ++q) used |= chosen[q] == f;
            const unsigned long long key = used ? 0ull : ordered(gains[f]);
            twice |= key != 0ull && key == bk;
            if (key > bk) {
                bk = key;
                bi = f;
                twice = false;
            }
        }
        const unsigned hi = static_cast<unsigned>(bk >> 32);
        const unsigned th = __reduce_max_sync(0xffffffffu, hi);
        const unsigned lo = hi == th ? static_cast<unsigned>(bk) : 0u;
        const unsigned tl = __reduce_max_sync(0xffffffffu, lo);
        const bool best = hi == th && lo == tl && bi != 0x7fffffff;
        const unsigned at = __ballot_sync(0xffffffffu, best);
        plain &= __popc(at) == 1 && !(best && twice);
        chosen[r] = __shfl_sync(0xffffffffu, bi, at ? __ffs(at) - 1 : 0);
        if (lane == 0) top[r] = chosen[r];
    }
    if (!__all_sync(0xffffffffu, plain)) {
        if (lane == 0) {
            for (int f = 0; f < n_f; ++f) scratch[f] = static_cast<short>(f);
            libstdcxx_sort(scratch, n_f, [&](short a, short b) { return gains[a] > gains[b]; });
            for (int r = 0; r < k; ++r) top[r] = scratch[r];
        }
    }
    __syncwarp();
}

template <bool kVar>
__global__ void __launch_bounds__(kPairThreads, 2)
    wave_pair_kernel(const WaveCtx* __restrict__ ctxs, int n_ctx, int src) {
    constexpr int kPlanes = kVar ? 5 : 3;  // g low, g high, (h low, h high,) counts
    constexpr int kCells = kMaxPairs * kBins;
    extern __shared__ __align__(16) unsigned int s_pl[];  // [kPlanes][kCells]
    __shared__ WaveCtx s_ctx;
    __shared__ int s_pref[kMaxWaveCtx + 1];
    __shared__ int s_count[kPairThreads], s_chunk0[kPairThreads + 1], s_wsum[kPairWarps];
    __shared__ double s_gains[kMaxPairFeatures];
    __shared__ short s_sort[kMaxPairFeatures];
    __shared__ int s_top[kPairTop], s_last;
    __shared__ Cand s_best[kMaxPairs];
    stage_ctx(s_ctx, ctxs);
    for (int q = threadIdx.x; q < kPlanes * kCells / 4; q += kPairThreads)
        reinterpret_cast<uint4*>(s_pl)[q] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    auto ctx_of = [&](int c) -> const WaveCtx& { return c == 0 ? s_ctx : ctxs[c]; };
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    children_prefix(ctxs, n_ctx, src, s_pref);
    const int total = s_pref[n_ctx];
    for (int j0 = 0; j0 < total; j0 += kPairThreads) {
        // a thread per child: its rows when it is weak
        int c = 0, cnt = 0;
        const int j = j0 + static_cast<int>(threadIdx.x);
        if (j < total) {
            while (c + 1 < n_ctx && s_pref[c + 1] <= j) ++c;
            const WaveCtx& X = ctx_of(c);
            if (X.pair_on) {
                const WaveChild t = scan_child(X, src, j - s_pref[c]);
                const DevNode* N = child_node(X, src, t.ci);
                const DevSplit* axis = child_split(X, src, t.ci);
                const double axis_gain = axis->valid ? axis->gain : -1e300;
                const double energy = static_cast<double>(X.energy[t.ci]) * ldexp(1.0, -energy_shift(X.st));
                const bool weak = t.eligible && X.gp.n_features >= 2 && X.pair_top_k >= 2 &&
                                  ((axis_gain < X.pair_trigger * fmax(energy * 0.01, 1e-12)) || axis_gain <= 0);
                if (weak) cnt = N->count;
                // no pair search: also for a weak child without rows (min_samples_leaf 0), which no chunk finishes
                if (cnt == 0 && j % static_cast<int>(gridDim.x) == static_cast<int>(blockIdx.x))
                    *(src == 0 ? X.splits_pair : X.spec_split_pair + t.ci) = *axis;
            }
        }
        // chunks of the batch's weak children
        int sum = cnt;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        __syncthreads();  // the previous batch is done
        if (lane == 0) s_wsum[warp] = sum;
        s_count[threadIdx.x] = cnt;
        __syncthreads();
        long long all = 0;
#pragma unroll
        for (int w = 0; w < kPairWarps; ++w) all += s_wsum[w];
        if (all == 0) continue;
        const long long per = (all + gridDim.x - 1) / gridDim.x;
        const int chunk = static_cast<int>(
            min(static_cast<long long>(kPairChunk), max(static_cast<long long>(kPairMinChunk), (per + 255) / 256 * 256)));
        const int nch = (cnt + chunk - 1) / chunk;
        int incl = nch;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        __syncthreads();  // every thread has read s_wsum
        if (lane == 31) s_wsum[warp] = incl;
        __syncthreads();
        int before = 0, tasks = 0;
#pragma unroll
        for (int w = 0; w < kPairWarps; ++w) {
            if (w < warp) before += s_wsum[w];
            tasks += s_wsum[w];
        }
        s_chunk0[threadIdx.x] = before + incl - nch;
        if (threadIdx.x == 0) s_chunk0[kPairThreads] = tasks;
        __syncthreads();
        for (int task = blockIdx.x; task < tasks; task += gridDim.x) {
            int lo = 0, hi = kPairThreads - 1;  // the last child that starts at or before the task
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (s_chunk0[mid] <= task) lo = mid;
                else hi = mid - 1;
            }
            const int jj = j0 + lo, n_chunks = s_chunk0[lo + 1] - s_chunk0[lo];
            int cc = 0;
            while (cc + 1 < n_ctx && s_pref[cc + 1] <= jj) ++cc;
            const WaveCtx& X = ctx_of(cc);
            const GrowParams& p = X.gp;
            const int k_child = jj - s_pref[cc], n_f = p.n_features;
            const WaveChild t = scan_child(X, src, k_child);
            const DevNode* N = child_node(X, src, t.ci);
            const int buf = N->buf, start = N->start;
            const int k = min(min(X.pair_top_k, kPairTop), n_f), n_pairs = k * (k - 1) / 2;
            for (int f = threadIdx.x; f < n_f; f += kPairThreads)
                s_gains[f] = X.cand_gain[static_cast<size_t>(t.ci) * n_f + f];
            __syncthreads();
            if (warp == 0) top_features(s_gains, n_f, k, s_sort, s_top);
            __syncthreads();
            const uint8_t* col[kPairTop];
#pragma unroll
            for (int a = 0; a < kPairTop; ++a)
                col[a] = X.codes_col + static_cast<size_t>(s_top[a < k ? a : 0]) * X.col_pitch;
            const int32_t* rows = (buf ? X.rows1 : X.rows0) + start;
            const long long pos0 = static_cast<long long>(buf) * X.pay_pitch + start;
            const long long* gpay = static_cast<const long long*>(X.gq) + pos0;
            const long long* hpay = kVar ? static_cast<const long long*>(X.hq) + pos0 : nullptr;
            // x mod n_bins for 32-bit x: the quotient by floor(2^32 / n_bins) is at most one short
            const unsigned nb = static_cast<unsigned>(p.n_bins);
            const unsigned inv = nb > 1u ? static_cast<unsigned>(0x100000000ull / nb) : 0u;
            const int r0 = (task - s_chunk0[lo]) * chunk, r1 = min(s_count[lo], r0 + chunk);
            for (int i = r0 + static_cast<int>(threadIdx.x); i < r1; i += kPairThreads) {
                const int r = rows[i];
                const long long gv = gpay[i];
                const long long hv = kVar ? hpay[i] : 0;
                unsigned cd[kPairTop];
#pragma unroll
                for (int a = 0; a < kPairTop; ++a) cd[a] = a < k ? col[a][r] : 0u;
                const long long v = kVar ? gv : gv >> 1;
                const unsigned g_lo = static_cast<unsigned>(v) & ((1u << kPairLo) - 1u);
                const unsigned g_hi = static_cast<unsigned>(static_cast<int>(v >> kPairLo));
                const unsigned h_lo = static_cast<unsigned>(hv) & ((1u << kPairLo) - 1u);
                const unsigned h_hi = static_cast<unsigned>(static_cast<int>(hv >> kPairLo));
                const unsigned one = kVar ? 1u : (gv & 1) ? 0x10000u : 1u;
                unsigned* P = s_pl;
#pragma unroll
                for (int a = 0; a < kPairTop; ++a)
#pragma unroll
                    for (int b = a + 1; b < kPairTop; ++b) {
                        if (b >= k) continue;
                        const unsigned x = cd[a] * 2654435761u + cd[b] * 40503u;  // pair_bin
                        unsigned z = x - __umulhi(x, inv) * nb;
                        if (z >= nb) z -= nb;
                        if (nb == 1u) z = 0u;
                        atomicAdd(&P[z], g_lo);
                        atomicAdd(&P[kCells + z], g_hi);
                        if constexpr (kVar) {
                            atomicAdd(&P[2 * kCells + z], h_lo);
                            atomicAdd(&P[3 * kCells + z], h_hi);
                        }
                        atomicAdd(&P[(kPlanes - 1) * kCells + z], one);
                        P += kBins;
                    }
            }
            __syncthreads();
            // add the chunk to the child's sums and clear the planes
            const unsigned long long hq1 = static_cast<unsigned long long>(__double2ll_rn(1.0 * X.st->hscale));
            const unsigned long long hq2 =
                static_cast<unsigned long long>(__double2ll_rn(1.0 * X.goss_scale * X.st->hscale));
            const size_t base = static_cast<size_t>(k_child) * kCells;
            for (int q = threadIdx.x; q < n_pairs * kBins; q += kPairThreads) {
                const unsigned cn = s_pl[(kPlanes - 1) * kCells + q];
                if (cn == 0u) continue;
                const long long gs = static_cast<long long>(static_cast<int>(s_pl[kCells + q])) * (1ll << kPairLo) + s_pl[q];
                unsigned long long hs;
                unsigned n = cn;
                if constexpr (kVar) {
                    hs = static_cast<unsigned long long>(
                        static_cast<long long>(static_cast<int>(s_pl[3 * kCells + q])) * (1ll << kPairLo) + s_pl[2 * kCells + q]);
                } else {
                    hs = static_cast<unsigned long long>(cn & 0xffffu) * hq1 + static_cast<unsigned long long>(cn >> 16) * hq2;
                    n = (cn & 0xffffu) + (cn >> 16);
                }
                atomicAdd(&X.pair_G[base + q], static_cast<unsigned long long>(gs));
                atomicAdd(&X.pair_H[base + q], hs);
                atomicAdd(&X.pair_C[base + q], static_cast<int>(n));
#pragma unroll
                for (int pl = 0; pl < kPlanes; ++pl) s_pl[pl * kCells + q] = 0u;
            }
            __threadfence();
            __syncthreads();
            if (threadIdx.x == 0) {
                s_last = atomicAdd(&X.pair_tickets[t.ci], 1) == n_chunks - 1;
                __threadfence();
            }
            __syncthreads();
            if (!s_last) continue;
            // the child's last chunk: scan the pairs, a warp each
            for (int q = warp; q < n_pairs; q += kPairWarps) {
                const size_t o = base + static_cast<size_t>(q) * kBins;
                long long Gt, Ht, Ct;
                const Cand cd =
                    scan_feature_warp(reinterpret_cast<long long*>(X.pair_G) + o, reinterpret_cast<long long*>(X.pair_H) + o,
                                      X.pair_C + o, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, false, true, 0,
                                      p.n_bins, X.st->inv_gscale, X.st->inv_hscale, X.pair_l2, p.min_split_gain,
                                      p.min_samples_leaf, p.min_child_weight, Gt, Ht, Ct);
                if (lane == 0) s_best[q] = cd;
            }
            __syncthreads();
            for (int q = threadIdx.x; q < n_pairs * kBins; q += kPairThreads) {
                X.pair_G[base + q] = 0ull;
                X.pair_H[base + q] = 0ull;
                X.pair_C[base + q] = 0;
            }
            if (threadIdx.x == 0) {
                const DevSplit axis = *child_split(X, src, t.ci);
                DevSplit best = axis;
                double bg = axis.valid ? axis.gain : -1e300;
                int q = 0;
                for (int a = 0; a < k; ++a)
                    for (int b = a + 1; b < k; ++b, ++q) {
                        const Cand cd = s_best[q];
                        if (cd.key == 0x7fffffff || !(cd.gain > bg)) continue;
                        bg = cd.gain;
                        best = DevSplit{};
                        best.gain = cd.gain;
                        best.valid = cd.gain >= p.min_split_gain;
                        best.feature = s_top[a];
                        best.feature2 = s_top[b];
                        best.type = 1;
                        best.threshold = (cd.key % 512) / 2;
                        best.missing_left = cd.key & 1;
                    }
                *(src == 0 ? X.splits_pair : X.spec_split_pair + t.ci) = best;
                X.pair_tickets[t.ci] = 0;
            }
            __syncthreads();  // shared state reuse
        }
    }
}

constexpr size_t pair_smem(bool var) { return static_cast<size_t>(var ? 5 : 3) * kMaxPairs * kBins * 4; }

}  // namespace

void prepare_wave_pair() {
    check(cudaFuncSetAttribute(wave_pair_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(pair_smem(false))), "wave_pair smem attr");
    check(cudaFuncSetAttribute(wave_pair_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(pair_smem(true))), "wave_pair smem attr");
}

void launch_wave_pair(const WaveCtx* ctxs, int n_ctx, int src, bool var, cudaStream_t s) {
    const dim3 grid(148 * 2);  // co-resident by registers
    if (var)
        launch_pdl(wave_pair_kernel<true>, grid, dim3(kPairThreads), pair_smem(true), s, "wave_pair launch", ctxs, n_ctx, src);
    else
        launch_pdl(wave_pair_kernel<false>, grid, dim3(kPairThreads), pair_smem(false), s, "wave_pair launch", ctxs, n_ctx,
                   src);
}

void launch_wave_scan(const WaveCtx* ctxs, int n_ctx, int src, int max_f, int ys, bool any_cat, cudaStream_t s) {
    launch_pdl(wave_scan_warp_kernel, dim3(148 * kScanWarpCtas), dim3(kScanWarpThreads), 0, s, "wave_scan launch", ctxs, n_ctx,
               src);
    if (any_cat)
        launch_pdl(wave_scan_cat_kernel, dim3(max_f, ys), dim3(kScanThreads), 0, s, "wave_scan_cat launch", ctxs, n_ctx,
                   src);
}

void launch_wave_select(const WaveCtx* ctxs, int n_ctx, int* gsync, unsigned* host_flag, unsigned long long cond,
                        int use_cond, cudaStream_t s) {
    launch_pdl(wave_select_kernel, dim3(n_ctx), dim3(kSelectThreads), 0, s, "wave_select launch", ctxs, n_ctx, gsync,
               host_flag,
               static_cast<cudaGraphConditionalHandle>(cond), use_cond);
}

}  // namespace tgb
