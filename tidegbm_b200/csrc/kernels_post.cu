// Per-tree sweep over all rows after a tree is grown.  Restates
// Booster::fit's grow_head tail (cpp/src/booster.cpp:589-664):
//   apply_all (cpp/src/tree.cpp:43-55)           leaf id of every row
//   full-data leaf values                        leaf_value(sum g, sum h) over ALL rows,
//                                                unscaled g and h (booster.cpp:594-600)
//   TORB prefix values                           per time bucket b, leaf values from the
//                                                rows [0, cut_b) of its causal past,
//                                                blended toward the full value when the
//                                                past is short (booster.cpp:604-648)
//   prediction update                            pred += lr * prefix[bucket][leaf]
//                                                (booster.cpp:655-664)
//
// Rows are sorted by time, so every cut is a row position and the rows between two
// consecutive distinct cuts form a segment.  apply_accum sums (g, h, 1) per
// (segment, leaf) in exact 64-bit fixed point (one shift per tree from max |g|,
// max h over all rows); finalize turns segment sums into prefix sums per bucket.
// CTAs own segment-aligned row chunks, so each CTA accumulates into one segment in
// shared memory (32-bit atomics) and adds its totals to the segment with one global
// 64-bit atomic per leaf and value.
#include <atomic>
#include "tgb_internal.h"

namespace tgb {

namespace {

constexpr int kApplyThreads = 256;

__global__ void all_scale_finalize_kernel(AllScale* sc, int n) { finalize_all_scale(sc, n); }

// Exact 64-bit add into (low, high) 32-bit shared words: the low word's returned old
// value says whether this addition wrapped; the carry goes to the high word.
__device__ __forceinline__ void add64s(unsigned int* lo, unsigned int* hi, int k, unsigned long long v) {
    const unsigned int vlo = static_cast<unsigned int>(v);
    const unsigned int old = atomicAdd(&lo[k], vlo);
    const unsigned int up = static_cast<unsigned int>(v >> 32) + (old + vlo < old ? 1u : 0u);
    if (up != 0u) atomicAdd(&hi[k], up);
}

constexpr int kApplyRows = 8;  // rows a thread walks together in the gather walk (two in the staged one)

// Staged walk: a block stages, per tile of kStageRows rows, only the columns the tree
// splits on (each distinct split feature once, 16-byte copies of whole tile runs) in shared
// memory and walks its rows there: a row costs one byte per distinct split feature
// instead of one 32-byte sector share per level.  Up to kMaxStaged / 2 columns leave room for
// two tiles, and the next one is copied while this one is walked.  A thread walks its two rows
// of a tile step by step together, over nodes of one 8-byte word each: a step is a chain of
// two shared loads and some ten instructions, and one row at a time left half of the issue
// slots empty.  10M rows, 31 leaves: 170 -> 107 us (their bytes take 55); 1.2M: 24 -> 18.  Trees over more than kMaxStaged distinct
// columns (or more than kMaxColWords * 32 features) take the gather walk: at each level
// the kApplyRows rows of a thread issue their column-major code loads together, and lanes
// at nodes with the same split feature share a sector.
constexpr int kStageRows = 512;
constexpr int kStagePitch = kStageRows + 16;  // a tile run starts up to 15 bytes early (16-byte loads)
constexpr int kMaxStaged = 64;
constexpr int kMaxColWords = 256;
constexpr size_t kApplySmem = static_cast<size_t>(kMaxStaged) * kStagePitch;

// kKinds: bit 0 the tree may hold categorical splits, bit 1 pair splits; a tree of axis
// splits only keeps neither the masks nor the second features in shared memory.
template <int kKinds>
__global__ void __launch_bounds__(kApplyThreads, 3)
    apply_accum_kernel(const uint8_t* __restrict__ col, long long pitch, int n_f, const DevNode* __restrict__ nodes,
                       const DevTreeState* __restrict__ st, const double* __restrict__ g,
                       const double* __restrict__ h, const int4* __restrict__ chunks,
                       int n_chunks, const AllScale* __restrict__ sc, int16_t* __restrict__ nid,
                       unsigned long long* __restrict__ seg_sums, int n_bins) {
    constexpr bool kCat = (kKinds & 1) != 0, kPair = (kKinds & 2) != 0;
    extern __shared__ __align__(16) uint8_t s_tile[];  // [kMaxStaged][kStagePitch]
    __shared__ int16_t s_feat[kMaxNodes], s_left[kMaxNodes], s_right[kMaxNodes];
    __shared__ uint8_t s_thr[kMaxNodes], s_ml[kMaxNodes], s_leaf[kMaxNodes], s_type[kMaxNodes];
    __shared__ int16_t s_feat2[kPair ? kMaxNodes : 1];
    __shared__ unsigned long long s_cat[kCat ? kMaxNodes : 1][4];  // left masks of categorical nodes
    __shared__ unsigned int s_bits[kMaxColWords];
    __shared__ int s_wbase[kMaxColWords], s_uf[kMaxStaged], s_nu;
    // Staged walk: a node in two words.  x: byte offset of its staged column 0-15; 16-24 and 25:
    // left iff code - bit 25 < bits 16-24 (unsigned; bit 25: missing goes right); split type
    // 26-27; leaf 31.  y: byte offsets of its children in this table 0-11 and 12-23 (a leaf's
    // are its own); second staged column 24-31.
    __shared__ uint2 s_word[kMaxNodes];
    // 64-bit sums as (low, high) 32-bit words: shared atomics stay single 32-bit operations.
    __shared__ unsigned int aGl[kMaxNodes], aGh[kMaxNodes], aHl[kMaxNodes], aHh[kMaxNodes], aC[kMaxNodes];
    const int nn = st->n_nodes;
    const int n_words = (n_f + 31) / 32;
    const bool can_stage = n_words <= kMaxColWords;
    if (can_stage)
        for (int w = threadIdx.x; w < n_words; w += blockDim.x) s_bits[w] = 0u;
    __syncthreads();
    for (int k = threadIdx.x; k < nn; k += blockDim.x) {
        const DevNode& N = nodes[k];
        s_feat[k] = static_cast<int16_t>(N.feature);
        s_left[k] = static_cast<int16_t>(N.left);
        s_right[k] = static_cast<int16_t>(N.right);
        s_thr[k] = static_cast<uint8_t>(N.threshold < 0 ? 0 : N.threshold);
        s_ml[k] = static_cast<uint8_t>(N.missing_left);
        s_type[k] = static_cast<uint8_t>(N.is_leaf ? 0 : N.type);
        if constexpr (kPair) s_feat2[k] = static_cast<int16_t>(!N.is_leaf && N.type == 1 ? N.feature2 : 0);
        if constexpr (kCat)
            for (int q = 0; q < 4; ++q) s_cat[k][q] = N.type == 2 ? N.cat[q] : 0ull;
        s_leaf[k] = static_cast<uint8_t>(N.is_leaf);
        aGl[k] = aGh[k] = aHl[k] = aHh[k] = aC[k] = 0u;
        if (can_stage && !N.is_leaf) {
            atomicOr(&s_bits[N.feature >> 5], 1u << (N.feature & 31));
            if (kPair && N.type == 1) atomicOr(&s_bits[N.feature2 >> 5], 1u << (N.feature2 & 31));
        }
    }
    __syncthreads();
    if (can_stage) {
        // distinct split columns: ranks by an exclusive prefix of the bitmap's popcounts
        if (threadIdx.x < 32) {
            const int lane = threadIdx.x;
            int run = 0;
            for (int w0 = 0; w0 < n_words; w0 += 32) {
                const int w = w0 + lane;
                const int c = w < n_words ? __popc(s_bits[w]) : 0;
                int incl = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += t;
                }
                if (w < n_words) s_wbase[w] = run + incl - c;
                run += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (lane == 0) s_nu = run;
        }
        __syncthreads();
        if (s_nu <= kMaxStaged) {
            for (int w = threadIdx.x; w < n_words; w += blockDim.x) {
                unsigned int bits = s_bits[w];
                int u = s_wbase[w];
                while (bits != 0u) {
                    s_uf[u++] = w * 32 + __ffs(bits) - 1;
                    bits &= bits - 1u;
                }
            }
            auto rank = [&](int f) {
                return s_wbase[f >> 5] + __popc(s_bits[f >> 5] & ((1u << (f & 31)) - 1u));
            };
            for (int k = threadIdx.x; k < nn; k += blockDim.x) {
                uint2 w;
                if (s_leaf[k]) {
                    w.x = 0x80000000u;
                    w.y = static_cast<unsigned>(k) * 8u | static_cast<unsigned>(k) * 8u << 12;
                } else {
                    const unsigned ml = s_ml[k] & 1u;
                    w.x = static_cast<unsigned>(rank(s_feat[k])) * kStagePitch | (s_thr[k] + ml) << 16 | (ml ^ 1u) << 25 |
                          (s_type[k] & 3u) << 26;
                    w.y = static_cast<unsigned>(s_left[k]) * 8u | static_cast<unsigned>(s_right[k]) * 8u << 12;
                    if constexpr (kPair)
                        if (s_type[k] == 1) w.y |= static_cast<unsigned>(rank(s_feat2[k])) << 24;
                }
                s_word[k] = w;
            }
        }
        __syncthreads();
    }
    const bool staged = can_stage && s_nu <= kMaxStaged;
    const double gs = sc->gscale, hs = sc->hscale;
    // unit hessians (h == nullptr): every row adds the same fixed-point 1, so H = count x that
    const unsigned long long h1 = static_cast<unsigned long long>(__double2ll_rn(1.0 * hs));
    const int nu = staged ? s_nu : 0;
    // the tile's columns: a warp per staged column, a lane per 16 bytes of its run
    auto stage = [&](int t0, int t1, uint8_t* tile) {
        const int a0 = t0 & ~15, n16 = (t1 - a0 + 15) >> 4;
        const int lane = threadIdx.x & 31;
        for (int u = threadIdx.x >> 5; u < nu; u += kApplyThreads / 32) {
            const uint8_t* src = col + static_cast<long long>(s_uf[u]) * pitch + a0;
            const unsigned dst = static_cast<unsigned>(__cvta_generic_to_shared(tile + u * kStagePitch));
            for (int v = lane; v < n16; v += 32)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * v), "l"(src + 16 * v) : "memory");
        }
    };
    auto step = [&](const uint8_t* trow, uint2& w, unsigned& at) {
        const unsigned int b = trow[w.x & 0xffffu];
        bool left = b - ((w.x >> 25) & 1u) < ((w.x >> 16) & 0x1ffu);
        if constexpr (kCat || kPair) {
            const int type = static_cast<int>(w.x >> 26) & 3;
            if (type != 0) {
                unsigned int b2 = 0u;
                if constexpr (kPair)
                    if (type == 1) b2 = trow[(w.y >> 24) * kStagePitch];
                const int k = static_cast<int>(at >> 3);
                left = goes_left(type, s_cat[kCat ? k : 0], s_thr[k], s_ml[k] != 0, b, b2, n_bins);
            }
        }
        at = (w.y >> (left ? 0 : 12)) & 0xfffu;
        w = *reinterpret_cast<const uint2*>(reinterpret_cast<const char*>(s_word) + at);
    };
    const bool two_tiles = 2 * nu <= kMaxStaged;
    uint8_t* tile = s_tile;
    if (staged && static_cast<int>(blockIdx.x) < n_chunks) {
        const int4 ch = chunks[blockIdx.x];
        stage(ch.y, min(ch.z, ch.y + kStageRows), tile);
    }
    // a CTA takes chunks in turn (the node tables above are staged once per CTA)
    for (int ci = blockIdx.x; ci < n_chunks; ci += gridDim.x) {
        const int4 ch = chunks[ci];  // {segment, row start, row end, unused}
        if (staged) {
            for (int t0 = ch.y; t0 < ch.z; t0 += kStageRows) {
                const int t1 = min(ch.z, t0 + kStageRows);
                // the next tile, of this chunk or the CTA's next
                int n0 = t0 + kStageRows, n1 = ch.z;
                if (n0 >= ch.z) {
                    n0 = n1 = 0;
                    if (ci + static_cast<int>(gridDim.x) < n_chunks) {
                        const int4 nx = chunks[ci + gridDim.x];
                        n0 = nx.y;
                        n1 = nx.z;
                    }
                }
                n1 = min(n1, n0 + kStageRows);
                static_assert(kStageRows == 2 * kApplyThreads, "two rows a thread");
                const int ra = t0 + threadIdx.x, rb = ra + kApplyThreads;
                const double ga = ra < t1 ? g[ra] : 0.0, gb = rb < t1 ? g[rb] : 0.0;
                const double ha = h != nullptr && ra < t1 ? h[ra] : 1.0, hb = h != nullptr && rb < t1 ? h[rb] : 1.0;
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncthreads();  // the tile is there, and the walks of the one before are done
                uint8_t* other = tile == s_tile ? s_tile + kMaxStaged / 2 * kStagePitch : s_tile;
                if (two_tiles && n0 < n1) stage(n0, n1, other);
                const uint8_t* trow = tile + (ra - (t0 & ~15));
                uint2 wa = s_word[0], wb = wa;
                unsigned ka = 0, kb = 0;
                if (ra >= t1) wa.x = 0x80000000u;
                if (rb >= t1) wb.x = 0x80000000u;
                while (static_cast<int>(wa.x & wb.x) >= 0) {
                    step(trow, wa, ka);
                    step(trow + kApplyThreads, wb, kb);
                }
                auto add = [&](int r, int k, double gv, double hv) {
                    nid[r] = static_cast<int16_t>(k);
                    add64s(aGl, aGh, k, static_cast<unsigned long long>(__double2ll_rn(gv * gs)));
                    if (h != nullptr) add64s(aHl, aHh, k, static_cast<unsigned long long>(__double2ll_rn(hv * hs)));
                    atomicAdd(&aC[k], 1u);
                };
                if (ra < t1) add(ra, static_cast<int>(ka >> 3), ga, ha);
                if (rb < t1) add(rb, static_cast<int>(kb >> 3), gb, hb);
                if (two_tiles) {
                    tile = other;
                } else if (n0 < n1) {
                    __syncthreads();  // this tile's walks are done
                    stage(n0, n1, tile);
                }
            }
        } else {
            for (int base = ch.y; base < ch.z; base += kApplyThreads * kApplyRows) {
                int r[kApplyRows], k[kApplyRows];
                double gv[kApplyRows], hv[kApplyRows];
    #pragma unroll
                for (int i = 0; i < kApplyRows; ++i) {
                    r[i] = base + threadIdx.x + i * kApplyThreads;
                    k[i] = 0;
                    const bool ok = r[i] < ch.z;
                    gv[i] = ok ? g[r[i]] : 0.0;  // loaded before the walk so their latency overlaps it
                    hv[i] = ok && h ? h[r[i]] : 1.0;
                    if (!ok) r[i] = -1;
                }
                for (int level = 0; level < kMaxNodes; ++level) {  // a path has fewer than kMaxNodes nodes
                    unsigned int b[kApplyRows], b2[kApplyRows];
                    bool any = false;
    #pragma unroll
                    for (int i = 0; i < kApplyRows; ++i) {
                        const bool walk = r[i] >= 0 && !s_leaf[k[i]];
                        b[i] = walk ? __ldg(col + static_cast<long long>(s_feat[k[i]]) * pitch + r[i]) : 0u;
                        if constexpr (kPair)
                            b2[i] = walk && s_type[k[i]] == 1
                                        ? __ldg(col + static_cast<long long>(s_feat2[k[i]]) * pitch + r[i])
                                        : 0u;
                        else
                            b2[i] = 0u;
                        any |= walk;
                    }
                    if (!any) break;
    #pragma unroll
                    for (int i = 0; i < kApplyRows; ++i) {
                        if (r[i] < 0 || s_leaf[k[i]]) continue;
                        bool left;
                        if constexpr (kCat || kPair)
                            left = goes_left(s_type[k[i]], s_cat[kCat ? k[i] : 0], s_thr[k[i]], s_ml[k[i]], b[i], b2[i],
                                             n_bins);
                        else
                            left = b[i] == 0u ? s_ml[k[i]] != 0 : static_cast<int>(b[i]) <= s_thr[k[i]];
                        k[i] = left ? s_left[k[i]] : s_right[k[i]];
                    }
                }
    #pragma unroll
                for (int i = 0; i < kApplyRows; ++i) {
                    if (r[i] < 0) continue;
                    nid[r[i]] = static_cast<int16_t>(k[i]);
                    add64s(aGl, aGh, k[i], static_cast<unsigned long long>(__double2ll_rn(gv[i] * gs)));
                    if (h != nullptr)
                        add64s(aHl, aHh, k[i], static_cast<unsigned long long>(__double2ll_rn(hv[i] * hs)));
                    atomicAdd(&aC[k[i]], 1u);
                }
            }
        }
        __syncthreads();
        unsigned long long* out = seg_sums + static_cast<size_t>(ch.x) * kMaxNodes * 3;
        for (int k = threadIdx.x; k < nn; k += blockDim.x) {
            if (aC[k] == 0u) continue;
            atomicAdd(out + 3 * k, (static_cast<unsigned long long>(aGh[k]) << 32) | aGl[k]);
            atomicAdd(out + 3 * k + 1, h != nullptr ? (static_cast<unsigned long long>(aHh[k]) << 32) | aHl[k]
                                                    : static_cast<unsigned long long>(aC[k]) * h1);
            atomicAdd(out + 3 * k + 2, static_cast<unsigned long long>(aC[k]));
            aGl[k] = aGh[k] = aHl[k] = aHh[k] = aC[k] = 0u;  // clear for the CTA's next chunk
        }
        __syncthreads();
    }
}

__device__ __forceinline__ double leaf_value(double G, double H, double l2) { return -G / (H + l2); }

// Leaf values, TORB prefixes and the tree's snapshot, one CTA.  A thread per node first runs over
// the segments and leaves the node's sums through each of them (in place), so that a bucket's
// prefix is one read; summing from the first segment for every (bucket, node) took 10 us at
// 32 buckets.  Then the maxima that the next tree's gradients and sample reduce into are reset.
__global__ void __launch_bounds__(1024)
    finalize_tree_kernel(PostParams pp, DevTreeState* __restrict__ st, unsigned long long* __restrict__ seg_sums,
                         const int* __restrict__ bucket_seg_end, const int* __restrict__ cuts, AllScale* __restrict__ sc,
                         const DevNode* __restrict__ nodes, TreeOut out) {
    pdl_wait();
    pdl_trigger();
    const int nn = st->n_nodes, t = st->tree, max_nodes = out.max_nodes;
    double* values = out.values + static_cast<size_t>(t) * max_nodes;
    int* cover = out.cover + static_cast<size_t>(t) * max_nodes;
    double* prefix = out.prefix + static_cast<size_t>(t) * out.n_buckets * max_nodes;
    DevNode* nodes_out = out.nodes + static_cast<size_t>(t) * max_nodes;
    const double ig = sc->inv_gscale, ih = sc->inv_hscale;
    for (int k = threadIdx.x; k < nn; k += blockDim.x) {
        unsigned long long G = 0, H = 0, Cn = 0;
#pragma unroll 8
        for (int s = 0; s < pp.n_segments; ++s) {
            unsigned long long* e = seg_sums + (static_cast<size_t>(s) * kMaxNodes + k) * 3;
            G += e[0];
            H += e[1];
            Cn += e[2];
            e[0] = G;
            e[1] = H;
        }
        values[k] = leaf_value(static_cast<double>(static_cast<long long>(G)) * ig,
                               static_cast<double>(static_cast<long long>(H)) * ih, pp.l2);
        cover[k] = static_cast<int>(Cn);
    }
    {
        // the tree as it was grown (16-byte words)
        const uint4* from = reinterpret_cast<const uint4*>(nodes);
        uint4* to = reinterpret_cast<uint4*>(nodes_out);
        for (int k = threadIdx.x; k < max_nodes * static_cast<int>(sizeof(DevNode) / 16); k += blockDim.x) to[k] = from[k];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        out.st[t] = *st;
        sc->maxg_bits = sc->maxh_bits = 0ull;
        st->max_abs_g_bits = st->max_h_bits = 0ull;
    }
    const int nb = pp.n_buckets;
    for (int q = threadIdx.x; q < nb * nn; q += blockDim.x) {
        const int b = q / nn, k = q % nn;
        const double full = values[k];
        double v;
        if (pp.iid_mode) {
            v = full;
        } else {
            long long pG = 0, pH = 0;
            const int end = bucket_seg_end[b];
            if (end > 0) {
                const unsigned long long* e = seg_sums + (static_cast<size_t>(end - 1) * kMaxNodes + k) * 3;
                pG = static_cast<long long>(e[0]);
                pH = static_cast<long long>(e[1]);
            }
            const double cov = static_cast<double>(cuts[b]);
            const double alpha = cov <= 0.0 ? 0.0 : fmin(1.0, cov / fmax(pp.min_cover, 1.0));
            const double pref = cov > 0.0 ? leaf_value(static_cast<double>(pG) * ig, static_cast<double>(pH) * ih, pp.l2)
                                          : full;
            v = alpha * pref + (1.0 - alpha) * full;
        }
        prefix[static_cast<size_t>(b) * nn + k] = v;
    }
}

__device__ __forceinline__ const double* tree_prefix(const TreeOut& out, int t) {
    return out.prefix + static_cast<size_t>(t) * out.n_buckets * out.max_nodes;
}

// time_buckets on time-sorted rows (cpp/src/booster.cpp:60-72): rank = row.
__device__ __forceinline__ int row_bucket(const PostParams& pp, int i) {
    if (pp.iid_mode) return 0;
    const int b = static_cast<int>(static_cast<double>(i) / max(pp.n, 1) * pp.n_buckets);
    return min(b, pp.n_buckets - 1);
}

// The prediction updates go over steps of kUpdRows rows a thread (256 apart), whose loads go out
// together.  The bucket is monotone in the row, so a step that starts and ends in one bucket, as
// nearly all do, divides twice and not once a row.  With the loss, 10M rows: 78 -> 52 us of a
// tree (its bytes take 52 at the copy rate), 1.2M: 20 -> 11.
constexpr int kUpdThreads = 256;
constexpr int kUpdRows = 4;
constexpr int kUpdStep = kUpdThreads * kUpdRows;

__global__ void __launch_bounds__(kUpdThreads)
    pred_update_kernel(PostParams pp, const int16_t* __restrict__ nid, TreeOut out,
                       const DevTreeState* __restrict__ st, double* __restrict__ pred) {
    pdl_wait();
    pdl_trigger();
    const double* __restrict__ prefix = tree_prefix(out, st->tree);
    const int nn = st->n_nodes;
    const int n = pp.n;
    for (long long base = static_cast<long long>(blockIdx.x) * kUpdStep; base < n;
         base += static_cast<long long>(gridDim.x) * kUpdStep) {
        const int i0 = static_cast<int>(base) + threadIdx.x;
        const int end = static_cast<int>(min(base + kUpdStep, static_cast<long long>(n)));
        double p[kUpdRows];
        int k[kUpdRows];
#pragma unroll
        for (int q = 0; q < kUpdRows; ++q) {
            const int i = i0 + q * kUpdThreads;
            p[q] = i < end ? pred[i] : 0.0;
            k[q] = i < end ? nid[i] : 0;
        }
        const int b0 = row_bucket(pp, static_cast<int>(base)), b1 = row_bucket(pp, end - 1);
#pragma unroll
        for (int q = 0; q < kUpdRows; ++q) {
            const int i = i0 + q * kUpdThreads;
            if (i >= end) continue;
            const int b = b0 == b1 ? b0 : row_bucket(pp, i);
            pred[i] = p[q] + pp.learning_rate * prefix[static_cast<size_t>(b) * nn + k[q]];
        }
    }
}

// pred update fused with the MSE training loss on the updated predictions
// (booster.cpp:655-664 then 704-706): per-block partial sums of (pred - y)^2.
// Also the next tree's mse gradient g = 1 * (pred - y) (objective.cpp:105-118,
// the same double the gradient kernel computes) and its largest |g| into sc (reset by
// finalize_tree), so that the next tree needs no separate pass over pred and y.  The last CTA to
// finish adds the partial sums up, in a fixed order, and writes the loss.
__global__ void __launch_bounds__(kUpdThreads)
    pred_update_loss_kernel(PostParams pp, const int16_t* __restrict__ nid, TreeOut out, DevTreeState* __restrict__ st,
                            double* __restrict__ pred, const double* __restrict__ y, double* __restrict__ partials,
                            double* __restrict__ g, AllScale* __restrict__ sc, int* __restrict__ ticket) {
    pdl_wait();
    pdl_trigger();
    const int t = st->tree;
    const double* __restrict__ prefix = tree_prefix(out, t);
    const int nn = st->n_nodes;
    const int n = pp.n;
    double acc = 0.0, mg = 0.0;
    for (long long base = static_cast<long long>(blockIdx.x) * kUpdStep; base < n;
         base += static_cast<long long>(gridDim.x) * kUpdStep) {
        const int i0 = static_cast<int>(base) + threadIdx.x;
        const int end = static_cast<int>(min(base + kUpdStep, static_cast<long long>(n)));
        double p[kUpdRows], yv[kUpdRows];
        int k[kUpdRows];
#pragma unroll
        for (int q = 0; q < kUpdRows; ++q) {
            const int i = i0 + q * kUpdThreads;
            p[q] = i < end ? pred[i] : 0.0;
            yv[q] = i < end ? y[i] : 0.0;
            k[q] = i < end ? nid[i] : 0;
        }
        const int b0 = row_bucket(pp, static_cast<int>(base)), b1 = row_bucket(pp, end - 1);
#pragma unroll
        for (int q = 0; q < kUpdRows; ++q) {
            const int i = i0 + q * kUpdThreads;
            if (i >= end) continue;
            const int b = b0 == b1 ? b0 : row_bucket(pp, i);
            const double pn = p[q] + pp.learning_rate * prefix[static_cast<size_t>(b) * nn + k[q]];
            pred[i] = pn;
            const double d = pn - yv[q];
            acc += 1.0 * d * d;
            const double gv = 1.0 * d;
            g[i] = gv;
            mg = fmax(mg, fabs(gv));
        }
    }
    block_max_into(mg, 1.0, sc);
    __shared__ double ws[32];
    __shared__ int s_last;
    auto block_sum = [&](double v) {
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = v;
        __syncthreads();
        double t = 0.0;
        for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) t += ws[w];
        __syncthreads();
        return t;
    };
    const double mine = block_sum(acc);
    if (threadIdx.x == 0) {
        partials[blockIdx.x] = mine;
        __threadfence();
        s_last = atomicAdd(ticket, 1) == static_cast<int>(gridDim.x) - 1;
        __threadfence();
    }
    __syncthreads();
    if (!s_last) return;
    double all = 0.0;
    for (int k = threadIdx.x; k < static_cast<int>(gridDim.x); k += blockDim.x) all += __ldcg(partials + k);
    all = block_sum(all);
    if (threadIdx.x == 0) {
        out.losses[t] = n > 0 ? all / static_cast<double>(n) : 0.0;
        *ticket = 0;
        st->tree = t + 1;  // every CTA has read it
    }
}

__global__ void fill_pred_kernel(const double* __restrict__ init_prefix, int n, int n_buckets, int iid_mode,
                                 double* __restrict__ pred) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        int b = 0;
        if (!iid_mode) {
            b = static_cast<int>(static_cast<double>(i) / max(n, 1) * n_buckets);
            if (b >= n_buckets) b = n_buckets - 1;
        }
        pred[i] = init_prefix[b];
    }
}

// Booster::predict_raw_binned (cpp/src/booster.cpp:744-773): base + sum over trees of
// lr * values[leaf], accumulated per row in tree order.
//
// Trees pass through shared memory in batches (at most kPredNodes nodes and kPredTrees
// trees): a node is one 64-bit word, a leaf's word points to itself, so a walk is a fixed
// number of steps without a test, and a lane walks four trees side by side (each step is two
// dependent shared loads).  A CTA of 8 warps takes RW x 32 rows, whose codes it stages with
// a pitch of an odd number of words (the lanes' rows start in different banks).  With RW < 8
// the batch's trees are split over 8 / RW warps, which leave their leaf values in shared memory
// for one warp to add up in tree order: few rows still fill the chip.  (One thread per row
// walking every tree through global memory took 217 us for 1,000 rows x 80 trees and
// 3,577 us for 1M x 200: four dependent loads a step and nothing else in flight; the whole
// calls went from 388 to 83 us and from 9.7 to 5.2 ms, of which the upload is 4.6.)
constexpr int kPredThreads = 256;
constexpr int kPredNodes = 2048;
constexpr int kPredTrees = 32;
constexpr int kPredWays = 4;
constexpr size_t kPredTable = static_cast<size_t>(kPredNodes) * 16;
constexpr size_t kPredMaxSmem = 200 * 1024;

// kVariant 0: axis splits only; 1: any split; 2: any split, codes read from global memory.
template <int RW, int kVariant>
__global__ void __launch_bounds__(kPredThreads)
    predict_trees_kernel(const uint8_t* __restrict__ codes, int stride, int n, const unsigned long long* __restrict__ word,
                         const double* __restrict__ val, const int4* __restrict__ trees,
                         const int* __restrict__ batches, int n_batches, double base, double lr,
                         const unsigned long long* __restrict__ cat, const int16_t* __restrict__ feat2, int n_bins,
                         double* __restrict__ out) {
    constexpr int TW = 8 / RW;
    extern __shared__ __align__(16) unsigned char s_raw[];
    unsigned long long* s_word = reinterpret_cast<unsigned long long*>(s_raw);
    double* s_val = reinterpret_cast<double*>(s_raw + kPredNodes * 8);
    double* s_leaf = reinterpret_cast<double*>(s_raw + kPredTable);  // TW > 1: [kPredTrees][32 RW]
    uint8_t* s_codes = s_raw + kPredTable + (TW > 1 ? kPredTrees * 32 * RW * 8 : 0);
    __shared__ int4 s_tree[kPredTrees];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rw = warp % RW, tw = warp / RW;
    const int row0 = blockIdx.x * 32 * RW, row = row0 + rw * 32 + lane;
    const int pitch = stride + 4;
    if (kVariant != 2) {
        const int per = stride / 16, here = min(32 * RW, n - row0);
        for (int q = threadIdx.x; q < here * per; q += kPredThreads) {
            const int r = q / per, k = q - r * per;
            const uint4 v = *reinterpret_cast<const uint4*>(codes + static_cast<size_t>(row0 + r) * stride + 16 * k);
            unsigned int* d = reinterpret_cast<unsigned int*>(s_codes + r * pitch + 16 * k);
            d[0] = v.x;
            d[1] = v.y;
            d[2] = v.z;
            d[3] = v.w;
        }
    }
    const uint8_t* mine =
        kVariant == 2 ? codes + static_cast<size_t>(min(row, n - 1)) * stride : s_codes + (rw * 32 + lane) * pitch;
    double s = base;
    for (int b = 0; b < n_batches; ++b) {
        const int t0 = batches[b], nt = batches[b + 1] - t0;
        __syncthreads();  // the previous batch is done (first: nothing is staged yet)
        if (static_cast<int>(threadIdx.x) < nt) s_tree[threadIdx.x] = trees[t0 + threadIdx.x];
        const int first = trees[t0].x, last = trees[t0 + nt - 1].x + trees[t0 + nt - 1].y;
        for (int k = threadIdx.x; k < last - first; k += kPredThreads) {
            s_word[k] = word[first + k];
            s_val[k] = val[first + k];
        }
        __syncthreads();
        const int share = (nt + TW - 1) / TW;
        const int a0 = min(nt, tw * share), a1 = min(nt, a0 + share);
        for (int a = a0; a < a1; a += kPredWays) {
            int k[kPredWays], o[kPredWays], depth = 0;
#pragma unroll
            for (int q = 0; q < kPredWays; ++q) {
                const int4 t = s_tree[min(a + q, a1 - 1)];  // {first node, nodes, depth, 0}
                o[q] = t.x - first;
                depth = max(depth, t.z);
                k[q] = 0;
            }
            for (int d = 0; d < depth; ++d) {
                unsigned long long w[kPredWays];
                unsigned int c[kPredWays];
#pragma unroll
                for (int q = 0; q < kPredWays; ++q) w[q] = s_word[o[q] + k[q]];
#pragma unroll
                for (int q = 0; q < kPredWays; ++q) c[q] = mine[static_cast<unsigned>(w[q] >> 40) & 0xffffu];
#pragma unroll
                for (int q = 0; q < kPredWays; ++q) {
                    const unsigned thr = static_cast<unsigned>(w[q] >> 32) & 0xffu;
                    const bool ml = (w[q] >> 56) & 1ull;
                    bool left = c[q] == 0u ? ml : c[q] <= thr;
                    if (kVariant != 0) {
                        const int type = static_cast<int>(w[q] >> 57) & 3;
                        if (type != 0) {
                            const size_t at = static_cast<size_t>(first + o[q] + k[q]);
                            const unsigned c2 = type == 1 ? mine[feat2[at]] : 0u;
                            left = goes_left(type, cat + 4 * at, static_cast<int>(thr), ml, c[q], c2, n_bins);
                        }
                    }
                    k[q] = static_cast<int>(static_cast<unsigned>(left ? w[q] : w[q] >> 16) & 0xffffu);
                }
            }
#pragma unroll
            for (int q = 0; q < kPredWays; ++q) {
                if (a + q >= a1) continue;
                const double v = s_val[o[q] + k[q]];
                if constexpr (TW == 1) s += lr * v;
                else s_leaf[(a + q) * 32 * RW + rw * 32 + lane] = v;
            }
        }
        if constexpr (TW > 1) {
            __syncthreads();
            if (tw == 0)
                for (int t = 0; t < nt; ++t) s += lr * s_leaf[t * 32 * RW + rw * 32 + lane];
        }
    }
    if (tw == 0 && row < n) out[row] = s;
}

template <int RW>
void predict_launch(int variant, size_t smem, const uint8_t* codes, int stride, int n, const PredictTrees& m, double base,
                    double lr, double* out, cudaStream_t s) {
    auto kern = variant == 0 ? predict_trees_kernel<RW, 0> : variant == 1 ? predict_trees_kernel<RW, 1>
                                                                          : predict_trees_kernel<RW, 2>;
    {
        static std::atomic<bool> done[64][3] = {};
        int dev = 0;
        check(cudaGetDevice(&dev), "cudaGetDevice");
        if (dev < 0 || dev >= 64 || !done[dev][variant]) {
            check(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kPredMaxSmem)),
                  "predict smem attr");
            if (dev >= 0 && dev < 64) done[dev][variant] = true;
        }
    }
    kern<<<(n + 32 * RW - 1) / (32 * RW), kPredThreads, smem, s>>>(codes, stride, n, m.word, m.val, m.trees, m.batches,
                                                                  m.n_batches, base, lr, m.cat, m.feat2, m.n_bins, out);
    check(cudaGetLastError(), "predict_trees launch");
}

}  // namespace

void launch_fill_pred(const double* init_prefix, int n, int n_buckets, int iid_mode, double* pred,
                      cudaStream_t s) {
    fill_pred_kernel<<<std::max(1, std::min(2368, (n + 255) / 256)), 256, 0, s>>>(init_prefix, n, n_buckets,
                                                                                  iid_mode, pred);
    check(cudaGetLastError(), "fill_pred launch");
}

int predict_batch_nodes() { return kPredNodes; }
int predict_batch_trees() { return kPredTrees; }

void launch_predict_trees(const uint8_t* codes, int stride, int n, const PredictTrees& m, double base, double lr,
                          double* out, cudaStream_t s) {
    if (n <= 0) return;
    // Rows a CTA: 256 once they fill two CTAs a SM (less staging of trees per row), else 128 or
    // 32 with the trees split over the warps; fewer where the rows' codes do not fit.  us by 32 / 128
    // / 256 rows, 32 features, 80 trees: 10,000 rows 13.3 / 15.2 / 26.7, 18,944 17.3 / 15.6 / 27.0,
    // 40,000 33.5 / 32.0 / 41.3, 75,776 57.0 / 43.0 / 42.3, 100,000 74.0 / 60.9 / 60.4.
    const size_t pitch = static_cast<size_t>(stride) + 4;
    auto smem = [&](int rw) {
        return kPredTable + (rw < 8 ? static_cast<size_t>(kPredTrees) * 32 * rw * 8 : 0) + pitch * 32 * rw;
    };
    int rw = n >= 148 * 2 * 256 ? 8 : n >= 148 * 128 ? 4 : 1;
    while (rw > 1 && smem(rw) > kPredMaxSmem) rw = rw == 8 ? 4 : 1;
    int variant = m.any_kind ? 1 : 0;
    size_t bytes = smem(rw);
    if (bytes > kPredMaxSmem) {
        variant = 2;
        bytes -= pitch * 32 * rw;
    }
    if (rw == 8) predict_launch<8>(variant, bytes, codes, stride, n, m, base, lr, out, s);
    else if (rw == 4) predict_launch<4>(variant, bytes, codes, stride, n, m, base, lr, out, s);
    else predict_launch<1>(variant, bytes, codes, stride, n, m, base, lr, out, s);
}

// Four CTAs an SM at most: a CTA's reductions cost more than its rows on small data.
int pred_update_parts(int n) {
    return static_cast<int>(std::max(1ll, std::min(592ll, (static_cast<long long>(n) + kUpdStep - 1) / kUpdStep)));
}

void launch_pred_update_loss(const PostParams& pp, const int16_t* nid, const TreeOut& out, DevTreeState* st,
                             double* pred, const double* y, double* partials, double* g, AllScale* sc, int* ticket,
                             cudaStream_t s) {
    launch_pdl(pred_update_loss_kernel, dim3(pred_update_parts(pp.n)), dim3(kUpdThreads), 0, s, "pred_update_loss launch", pp, nid,
               out, st, pred, y, partials, g, sc, ticket);
}

void launch_all_scale_finalize(AllScale* sc, int n, cudaStream_t s) {
    all_scale_finalize_kernel<<<1, 1, 0, s>>>(sc, n);
    check(cudaGetLastError(), "all_scale_finalize launch");
}

void launch_apply_accum(const uint8_t* col, long long pitch, int n_f, const DevNode* nodes, const DevTreeState* st,
                        const double* g, const double* h, const int4* chunks, int n_chunks,
                        const AllScale* sc, int16_t* nid, unsigned long long* seg_sums, int n_bins, int kinds,
                        cudaStream_t s) {
    auto kern = kinds == 0 ? apply_accum_kernel<0> : kinds == 1 ? apply_accum_kernel<1>
                                                   : kinds == 2 ? apply_accum_kernel<2> : apply_accum_kernel<3>;
    {  // static + dynamic shared memory above 48 KB needs the opt-in, once per device
        static std::atomic<bool> done[64][4] = {};
        int dev = 0;
        check(cudaGetDevice(&dev), "cudaGetDevice");
        if (dev < 0 || dev >= 64 || !done[dev][kinds & 3]) {
            check(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kApplySmem)),
                  "apply_accum smem attr");
            if (dev >= 0 && dev < 64) done[dev][kinds & 3] = true;
        }
    }
    // a persistent grid: 3 CTAs per SM (its register and shared-memory budget), chunks in turn
    int sms = 148;
    {
        int dev = 0;
        if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    }
    const int grid = std::max(1, std::min(n_chunks, 3 * sms));
    kern<<<grid, kApplyThreads, kApplySmem, s>>>(col, pitch, n_f, nodes, st, g, h, chunks, n_chunks, sc, nid,
                                                 seg_sums, n_bins);
    check(cudaGetLastError(), "apply_accum launch");
}

void launch_finalize_tree(const PostParams& pp, DevTreeState* st, unsigned long long* seg_sums,
                          const int* bucket_seg_end, const int* cuts, AllScale* sc, const DevNode* nodes,
                          const TreeOut& out, cudaStream_t s) {
    launch_pdl(finalize_tree_kernel, dim3(1), dim3(1024), 0, s, "finalize_tree launch", pp, st, seg_sums, bucket_seg_end,
               cuts, sc, nodes, out);
}

void launch_pred_update(const PostParams& pp, const int16_t* nid, const TreeOut& out, const DevTreeState* st,
                        double* pred, cudaStream_t s) {
    launch_pdl(pred_update_kernel, dim3(pred_update_parts(pp.n)), dim3(kUpdThreads), 0, s, "pred_update launch", pp, nid, out, st,
               pred);
}

}  // namespace tgb
