// Wave kernels: batched histograms and partitions over many leaves of many trees, and
// the per-tree set-up of a context (wave.h describes the scheme).
//
// Histogram (build_hist_col, cpp/src/histogram.cpp:44-76, for the smaller child of every
// planned leaf; subtract_hist_inplace's larger child is derived in the scan).  One
// persistent launch of clusters of 1, 2 or 4 CTAs (the autotuned privatisation depth:
// how many CTA-private histograms a flush merges).  The work (rows x groups of 32
// features, summed over the jobs) is cut into one range per cluster, walked as pieces
// (job, feature group, rows) whose rows the cluster's CTAs split.  Inside a CTA the
// accumulation is the lane-per-row scheme:
// a warp takes 32 rows, lane l holds its row's 32 code bytes of the group (staged in shared
// memory by TMA gathers in the constant-hessian modes, else loaded from global memory) and
// rotates them by l bytes in registers, so step j of the 32-step loop
// touches feature (j + l) & 31: 32 lanes, 32 features, 32 banks of the [bin][feature]
// layout, conflict-free whatever the codes.  Every code costs fire-and-forget 32-bit
// shared reductions only (their count depends on the payload mode, below), exact over a
// sub-chunk of rows, folded into 64-bit totals after every sub-chunk.  At the end of a
// piece the cluster adds its CTAs' totals through distributed shared memory and each CTA
// writes its share of the cells out (coalesced: consecutive bins of a feature).
//
// Payload modes (HistMode, per row):
//   exact const  int64 (v << 1 | goss):  v split into a 19-bit low and a signed high
//                part, plus a packed (unscaled, GOSS-scaled) row count: 3 reductions
//   exact var    int64 g and int64 h (both 19-bit split) and a count: 5 reductions
//   q16 const    int32 (q << 1 | goss): q and the packed count: 2 reductions
//   q16 var      int32 (qg << 16 | qh): qg, qh and a count: 3 reductions
//   q8 const     int16 (q << 1 | goss): (1 << 20 | q + 128) into the row class's
//                plane: 1 reduction
//   q8 var       uint16 (qg + 128 | qh << 8): (1 << 20 | qg + 128) and qh: 2 reductions
// Sums of quantised values are exact integers; the scan rescales them.
//
// Partition (split_indices, cpp/src/tree.cpp:68-91): one launch over 2048-row tiles of all
// planned leaves (in-tile ballot ranks; tiles reserve their places with one atomic).
#include <atomic>
#include <cstdint>
#include <cstring>
#include <cooperative_groups.h>

#include "wave.h"

namespace tgb {

namespace cg = cooperative_groups;

namespace {

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr int kFG = 32;
constexpr int kPlane = kFG * kBins;  // 32-bit words per plane (8192)
constexpr int kCells = kPlane / kThreads;  // cells a thread folds (8)
constexpr size_t kPlaneBytes = static_cast<size_t>(kPlane) * 4;
constexpr int kLoBits = 19;

template <int kMode>
struct ModeTraits;
template <>
struct ModeTraits<kHistExactConst> {
    static constexpr int planes = 3, sub = 8192;
    static constexpr bool var = false;
};
template <>
struct ModeTraits<kHistExactVar> {
    static constexpr int planes = 5, sub = 8192;
    static constexpr bool var = true;
};
template <>
struct ModeTraits<kHistQ16Const> {
    static constexpr int planes = 2, sub = 32768;
    static constexpr bool var = false;
};
template <>
struct ModeTraits<kHistQ16Var> {
    static constexpr int planes = 3, sub = 32768;
    static constexpr bool var = true;
};
template <>
struct ModeTraits<kHistQ8Const> {
    static constexpr int planes = 2, sub = 3072;
    static constexpr bool var = false;
};
template <>
struct ModeTraits<kHistQ8Var> {
    static constexpr int planes = 2, sub = 3072;
    static constexpr bool var = true;
};

// out[t] = in[(t + k) & 7] for a lane-dependent k in [0, 8): three conditional rotations.
__device__ __forceinline__ void rotate_words(unsigned int (&w)[8], int k) {
    unsigned int t[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) t[i] = (k & 1) ? w[(i + 1) & 7] : w[i];
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = (k & 2) ? t[(i + 2) & 7] : t[i];
#pragma unroll
    for (int i = 0; i < 8; ++i) t[i] = (k & 4) ? w[(i + 4) & 7] : w[i];
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = t[i];
}

// Rows of one histogram job: the root's sample or a planned leaf's smaller child.
struct JobRows {
    const int32_t* rows;
    const void* gq;  // payloads of rows[0 ..) (same positions)
    const void* hq;
    int count;
    int slot;
};

__device__ __forceinline__ int job_count(const WaveCtx& X, int src, int e) {
    return src == 0 ? X.st->n_sample : X.ctl->job[e].count;
}

__device__ __forceinline__ JobRows job_rows(const WaveCtx& X, int src, int e) {
    WaveJob j{0, 0, 0, 0};
    if (src == 0) j.count = X.st->n_sample;
    else j = X.ctl->job[e];
    JobRows r;
    r.rows = (j.buf ? X.rows1 : X.rows0) + j.start;
    const long long pos = static_cast<long long>(j.buf) * X.pay_pitch + j.start;
    r.gq = static_cast<const unsigned char*>(X.gq) + pos * X.pay_bytes;
    r.hq = X.hq != nullptr ? static_cast<const long long*>(X.hq) + pos : nullptr;
    r.count = j.count;
    r.slot = j.slot;
    return r;
}

// A row's 32 code bytes of a feature group: one 32-byte load where the row stride keeps it
// 32-byte aligned (two_chunks: the group has 32 bytes before the row's end), else two
// 16-byte loads (the second only when the group has 32 bytes).
__device__ __forceinline__ void load_codes(const uint8_t* p, bool v8, bool two_chunks, uint4& a, uint4& b) {
    if (v8) {
        asm volatile("ld.global.nc.v8.u32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
                     : "l"(p));
    } else {
        const uint4* p4 = reinterpret_cast<const uint4*>(p);
        a = __ldg(p4);
        b = two_chunks ? __ldg(p4 + 1) : make_uint4(0, 0, 0, 0);
    }
}

// A CTA's totals in a padded [feature][bin] layout, index f * kTotPitch + b: the fold
// writes one bin of a warp's 32 features and the flush reads 32 consecutive bins of one
// feature, and with a pitch of 257 words both touch 32 distinct banks; the flush's global
// writes are then consecutive bins of a feature (whole sectors).
constexpr int kTotPitch = kBins + 1;
constexpr int kTot = kFG * kTotPitch;  // 8224 cells
// Rows of one CTA's share of a piece: the constant-hessian modes pack their two row counts
// (unscaled, GOSS-scaled) into 16-bit halves.
constexpr int kMaxShareRows = 65535;

// Dynamic shared memory of one instantiation.  Constant-hessian modes: the working planes,
// then the totals (G as 64-bit words, packed counts), folded every sub-chunk.  Per-row
// hessian modes: 64-bit register accumulators, their totals (G, H as 64-bit words, counts)
// written over the working planes at the end of a piece.  Then the work prefix of the jobs.
template <int kMode>
struct SmemLayout {
    using T = ModeTraits<kMode>;
    static constexpr size_t work = static_cast<size_t>(T::planes) * kPlaneBytes;
    static constexpr size_t tot_bytes = static_cast<size_t>(kTot) * (T::var ? 20 : 12);
    static constexpr size_t tot_off = T::var ? 0 : work;
    static constexpr size_t region = T::var ? (work > tot_bytes ? work : tot_bytes) : work + tot_bytes;
    static constexpr size_t plan_off = (region + 15) / 16 * 16;
    static constexpr size_t bytes = plan_off + sizeof(unsigned long long) * (kMaxWaveJobs + 1);
    static_assert(bytes + 2048 <= 232448, "wave histogram shared memory above the 227 KB opt-in");
    static_assert(region % 16 == 0 && tot_off % 16 == 0, "16-byte zeroing");
};

template <int kMode>
struct ConstPayload;
template <>
struct ConstPayload<kHistExactConst> {
    using type = long long;
};
template <>
struct ConstPayload<kHistQ16Const> {
    using type = int;
};
template <>
struct ConstPayload<kHistQ8Const> {
    using type = short;
};

// One row of a constant-hessian mode: its 32 codes (two 16-byte words, rotated by the
// lane so that step j touches feature (j + lane) & 31) into the working planes.
template <int kMode>
__device__ __forceinline__ void add_row_const(unsigned int* __restrict__ P, typename ConstPayload<kMode>::type p,
                                              const uint4 ca, const uint4 cb, int lane, int q, int sh) {
    unsigned int a0, a1 = 0u, a2 = 0u;
    unsigned int* plane = P;
    if constexpr (kMode == kHistExactConst) {
        const long long v = p >> 1;
        a0 = static_cast<unsigned int>(v) & ((1u << kLoBits) - 1u);
        a1 = static_cast<unsigned int>(static_cast<int>(v >> kLoBits));
        a2 = (p & 1) ? 0x10000u : 1u;
    } else if constexpr (kMode == kHistQ16Const) {
        a0 = static_cast<unsigned int>(p >> 1);
        a1 = (p & 1) ? 0x10000u : 1u;
    } else {
        const int pv = p;
        a0 = (1u << 20) | static_cast<unsigned int>((pv >> 1) + 128);
        plane = (pv & 1) ? P + kPlane : P;
    }
    unsigned int wd[8] = {ca.x, ca.y, ca.z, ca.w, cb.x, cb.y, cb.z, cb.w};
    rotate_words(wd, q);
    unsigned int Rw[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) Rw[t] = __funnelshift_r(wd[t], wd[(t + 1) & 7], sh);
#pragma unroll
    for (int jj = 0; jj < 32; ++jj) {
        const int f = (jj + lane) & 31;
        const unsigned int code = (Rw[jj >> 2] >> ((jj & 3) * 8)) & 0xffu;
        const int cell = static_cast<int>(code) * 32 + f;
        if constexpr (kMode == kHistExactConst) {
            atomicAdd(&P[cell], a0);
            atomicAdd(&P[kPlane + cell], a1);
            atomicAdd(&P[2 * kPlane + cell], a2);
        } else if constexpr (kMode == kHistQ16Const) {
            atomicAdd(&P[cell], a0);
            atomicAdd(&P[kPlane + cell], a1);
        } else {
            atomicAdd(&plane[cell], a0);
        }
    }
}

// The rows [r0, r1) of a CTA's share of one piece (one group of 32 features), constant-
// hessian modes, lane = row: every code costs the mode's fire-and-forget 32-bit shared
// reductions, exact over a sub-chunk of rows and folded into the shared 64-bit totals after
// it.  Software-pipelined: a warp's next row index is loaded two steps ahead and its codes
// and payload one step ahead, so their latency overlaps the current step's reductions.  A
// separate (not inlined) function: the loop keeps only its own state in registers.
template <int kMode>
__device__ __noinline__ void accumulate_const(unsigned int* __restrict__ P, unsigned long long* __restrict__ Gt,
                                              unsigned int* __restrict__ Ct, const int32_t* __restrict__ rows, int r0,
                                              int r1, const uint8_t* __restrict__ codes, int stride, int fg0,
                                              const void* __restrict__ gqp) {
    using T = ModeTraits<kMode>;
    using PT = typename ConstPayload<kMode>::type;
    const PT* __restrict__ pay = static_cast<const PT*>(gqp);  // by position, like rows
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int q = lane >> 2, sh = (lane & 3) * 8;
    const bool two_chunks = stride - fg0 >= 32;
    const bool v8 = two_chunks && (stride & 31) == 0;
    constexpr int kStep = kWarps * 32;
    for (int k = threadIdx.x; k < kTot; k += kThreads) {
        Gt[k] = 0ull;
        Ct[k] = 0u;
    }
    __syncthreads();
    for (int s0 = r0; s0 < r1; s0 += T::sub) {
        const int s1 = min(r1, s0 + T::sub);
        const int k0 = s0 + warp * 32 + lane;
        int r_cur = k0 < s1 ? rows[k0] : -1;
        PT p = k0 < s1 ? pay[k0] : PT(0);
        int r_nxt = k0 + kStep < s1 ? rows[k0 + kStep] : -1;
        PT p_nxt = k0 + kStep < s1 ? pay[k0 + kStep] : PT(0);
        uint4 ca = make_uint4(0, 0, 0, 0), cb = make_uint4(0, 0, 0, 0);
        if (r_cur >= 0) load_codes(codes + static_cast<size_t>(r_cur) * stride + fg0, v8, two_chunks, ca, cb);
        for (int base = s0 + warp * 32; base < s1; base += kStep) {
            const int r = r_cur;
            const uint4 xa = ca, xb = cb;
            const PT xp = p;
            r_cur = r_nxt;
            p = p_nxt;
            const int kn = base + 2 * kStep + lane;
            r_nxt = kn < s1 ? rows[kn] : -1;
            p_nxt = kn < s1 ? pay[kn] : PT(0);
            if (r_cur >= 0) load_codes(codes + static_cast<size_t>(r_cur) * stride + fg0, v8, two_chunks, ca, cb);
            if (r >= 0) add_row_const<kMode>(P, xp, xa, xb, lane, q, sh);
        }
        __syncthreads();
        // fold the sub-chunk into the totals and clear the working planes
#pragma unroll
        for (int cc = 0; cc < kCells; ++cc) {
            const int cell = threadIdx.x + cc * kThreads;
            const int ti = (cell & 31) * kTotPitch + (cell >> 5);
            long long dg;
            unsigned int dc;
            if constexpr (kMode == kHistExactConst) {
                dg = static_cast<long long>(static_cast<int>(P[kPlane + cell])) * (1ll << kLoBits) + P[cell];
                dc = P[2 * kPlane + cell];
            } else if constexpr (kMode == kHistQ16Const) {
                dg = static_cast<int>(P[cell]);
                dc = P[kPlane + cell];
            } else {
                const unsigned int w1 = P[cell], w2 = P[kPlane + cell];
                const unsigned int n1 = w1 >> 20, n2 = w2 >> 20;
                dg = static_cast<long long>(w1 & 0xfffffu) + static_cast<long long>(w2 & 0xfffffu) -
                     128ll * static_cast<long long>(n1 + n2);
                dc = n1 | (n2 << 16);
            }
            Gt[ti] += static_cast<unsigned long long>(dg);
            Ct[ti] += dc;
#pragma unroll
            for (int pl = 0; pl < T::planes; ++pl) P[pl * kPlane + cell] = 0u;
        }
        __syncthreads();
    }
}

// ---- code rows staged by TMA (constant-hessian modes) ---------------------------------
// A warp owns two 1 KB staging slots (its batch of 32 rows x the group's 32 code bytes)
// and an mbarrier per slot.  Lanes 0-7 each gather four rows of a batch with one
// cp.async.bulk.tensor tile::gather4 (box: 32 bytes of one row), two batches ahead of the
// one the warp accumulates; a lane then reads its row from the slot with two conflict-free
// 16-byte shared loads.  The direct loads cost 32 scattered sectors per warp and row batch
// on the L1 data path that the shared reductions also use; the gathers leave it to them.
constexpr int kSlotBytes = 32 * kFG;                 // one warp's batch
constexpr int kSlotStride = kWarps * kSlotBytes;     // slot 1 of every warp after slot 0 of all
constexpr int kStageBytes = 2 * kSlotStride;         // 64 KB, over the 64-bit totals
constexpr int kSpinLimit = 1 << 18;                  // polls of one mbarrier wait
constexpr int kErrStaging = 3;                       // ctl->error: a staging wait gave up
static_assert(kStageBytes + 128 <= kTot * 8, "the staging slots lie inside the G totals");

__device__ __forceinline__ unsigned int smem_u32(const void* p) {
    return static_cast<unsigned int>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(unsigned int bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned int bar, unsigned int bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Polls phase `parity` of the barrier at most kSpinLimit times; false when it gave up.
__device__ __forceinline__ bool mbar_wait(unsigned int bar, unsigned int parity) {
    for (int it = 0; it < kSpinLimit; ++it) {
        unsigned int done;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}
// 16 bytes of shared memory at a 32-bit shared address (after the slot's barrier wait).
__device__ __forceinline__ uint4 lds16(unsigned int addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(addr)
                 : "memory");
    return v;
}
// Rows y0..y3, bytes [x, x + 32) of each, to dst (4 x 32 bytes), completing on bar.
__device__ __forceinline__ void tma_gather4(unsigned int dst, const CUtensorMap* map, int x, int y0, int y1, int y2,
                                            int y3, unsigned int bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst),
        "l"(map), "r"(x), "r"(y0), "r"(y1), "r"(y2), "r"(y3), "r"(bar)
        : "memory");
}

// accumulate_const with the code rows staged by TMA.  The 64-bit G totals are kept in
// registers (a thread owns the same cells as in the fold) and written to Gt at the end: the
// staging slots lie over Gt meanwhile; the counts fold into Ct as before.  `phase` holds the
// parity of each of the warp's two barriers across calls; returned updated.  A wait that
// gives up sets ctl->error and ends the staging for the rest of the call (no new gathers,
// no further waits but one bounded wait per gather still in flight).
template <int kMode>
__device__ __noinline__ unsigned int accumulate_const_tma(unsigned int* __restrict__ P,
                                                          unsigned long long* __restrict__ Gt,
                                                          unsigned int* __restrict__ Ct, unsigned char* stage,
                                                          unsigned long long* bars, unsigned int phase,
                                                          const int32_t* __restrict__ rows, int r0, int r1,
                                                          const CUtensorMap* map, int fg0,
                                                          const void* __restrict__ gqp, int* err) {
    using T = ModeTraits<kMode>;
    using PT = typename ConstPayload<kMode>::type;
    constexpr int kStep = kWarps * 32;
    constexpr int kFoldRounds = T::sub / kStep;
    static_assert(T::sub % kStep == 0, "a sub-chunk is whole rounds of the CTA");
    const PT* __restrict__ pay = static_cast<const PT*>(gqp);  // by position, like rows
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int q = lane >> 2, sh = (lane & 3) * 8;
    const unsigned int slot0 = smem_u32(stage) + warp * kSlotBytes;
    const unsigned int bar0 = smem_u32(bars + 2 * warp);
    long long accG[kCells];
#pragma unroll
    for (int cc = 0; cc < kCells; ++cc) accG[cc] = 0;
    // the staging area's generic writes (the previous piece's totals) before the gathers'
    // asynchronous ones
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    bool ok = true;
    unsigned int pending = 0u;  // slots with gathers in flight
    // The lane's row of batch k of this warp (the batch's first row pads a short batch),
    // loaded a round before its gather is issued.
    auto row_of = [&](int k) -> int {
        const int base = r0 + k * kStep + warp * 32;
        if (base >= r1) return 0;
        const int kk = base + lane;
        return rows[kk < r1 ? kk : base];
    };
    // Gathers batch k of this warp (lane rows `row`) into slot s; returns the lane's payload.
    auto issue = [&](int k, int s, int row) -> PT {
        const int base = r0 + k * kStep + warp * 32;
        if (!ok || base >= r1) return PT(0);
        const int kk = base + lane;
        const PT p = kk < r1 ? pay[kk] : PT(0);
        const int y0 = __shfl_sync(0xffffffffu, row, (4 * lane) & 31);
        const int y1 = __shfl_sync(0xffffffffu, row, (4 * lane + 1) & 31);
        const int y2 = __shfl_sync(0xffffffffu, row, (4 * lane + 2) & 31);
        const int y3 = __shfl_sync(0xffffffffu, row, (4 * lane + 3) & 31);
        const unsigned int bar = bar0 + 8u * s;
        if (lane == 0) mbar_expect_tx(bar, kSlotBytes);
        __syncwarp();
        if (lane < 8) tma_gather4(slot0 + s * kSlotStride + lane * 128, map, fg0, y0, y1, y2, y3, bar);
        pending |= 1u << s;
        return p;
    };
    const int n_rounds = r1 > r0 ? (r1 - r0 + kStep - 1) / kStep : 0;
    const int ra = row_of(0), rb = row_of(1);  // all three loads before the first use
    int rq = row_of(2);
    PT p0 = issue(0, 0, ra);
    PT p1 = issue(1, 1, rb);
    bool first = true;  // the first fold writes Ct, later ones add
    const int h = (lane >> 2) & 1;  // lanes 4-7 of each 8 read their second half first
    for (int i = 0; i < n_rounds; ++i) {
        const int s = i & 1;
        const int base = r0 + i * kStep + warp * 32;
        if (base < r1) {
            if (ok) {
                ok = __all_sync(0xffffffffu, mbar_wait(bar0 + 8u * s, (phase >> s) & 1u));
                if (ok) {
                    phase ^= 1u << s;
                    pending &= ~(1u << s);
                } else if (lane == 0) {
                    set_error(err, kErrStaging);
                }
            }
            const unsigned int rp = slot0 + s * kSlotStride + lane * 32;
            const uint4 c0 = lds16(rp + 16 * h);
            const uint4 c1 = lds16(rp + 16 * (h ^ 1));
            const uint4 ca = h ? c1 : c0, cb = h ? c0 : c1;
            const PT p = s ? p1 : p0;
            __syncwarp();  // every lane has read the slot before it is refilled
            const PT pn = issue(i + 2, s, rq);
            rq = row_of(i + 3);
            if (s) p1 = pn;
            else p0 = pn;
            if (base + lane < r1) add_row_const<kMode>(P, p, ca, cb, lane, q, sh);
        }
        if ((i + 1) % kFoldRounds == 0 || i + 1 == n_rounds) {
            __syncthreads();
            // fold the sub-chunk: G into registers, counts into Ct; clear the planes
#pragma unroll
            for (int cc = 0; cc < kCells; ++cc) {
                const int cell = threadIdx.x + cc * kThreads;
                const int ti = (cell & 31) * kTotPitch + (cell >> 5);
                long long dg;
                unsigned int dc;
                if constexpr (kMode == kHistExactConst) {
                    dg = static_cast<long long>(static_cast<int>(P[kPlane + cell])) * (1ll << kLoBits) + P[cell];
                    dc = P[2 * kPlane + cell];
                } else if constexpr (kMode == kHistQ16Const) {
                    dg = static_cast<int>(P[cell]);
                    dc = P[kPlane + cell];
                } else {
                    const unsigned int w1 = P[cell], w2 = P[kPlane + cell];
                    const unsigned int n1 = w1 >> 20, n2 = w2 >> 20;
                    dg = static_cast<long long>(w1 & 0xfffffu) + static_cast<long long>(w2 & 0xfffffu) -
                         128ll * static_cast<long long>(n1 + n2);
                    dc = n1 | (n2 << 16);
                }
                accG[cc] += dg;
                Ct[ti] = first ? dc : Ct[ti] + dc;
#pragma unroll
                for (int pl = 0; pl < T::planes; ++pl) P[pl * kPlane + cell] = 0u;
            }
            first = false;
            __syncthreads();
        }
    }
    if (!ok)  // warp-uniform
        for (int s = 0; s < 2; ++s)
            if (((pending >> s) & 1u) && __all_sync(0xffffffffu, mbar_wait(bar0 + 8u * s, (phase >> s) & 1u)))
                phase ^= 1u << s;
    // every warp is past its last slot read (the last round's fold): the totals over them
#pragma unroll
    for (int cc = 0; cc < kCells; ++cc) {
        const int cell = threadIdx.x + cc * kThreads;
        const int ti = (cell & 31) * kTotPitch + (cell >> 5);
        Gt[ti] = static_cast<unsigned long long>(accG[cc]);
        if (first) Ct[ti] = 0u;  // no rows
    }
    return phase;
}

// The rows [r0, r1) of a CTA's share of one piece, per-row hessian modes: the same lane-
// per-row reductions, folded into per-thread 64-bit registers every sub-chunk; the totals
// are written over the (then clear) working planes at the end.
template <int kMode>
__device__ __noinline__ void accumulate_var(unsigned int* __restrict__ P, unsigned long long* __restrict__ Gt,
                                            unsigned long long* __restrict__ Ht, unsigned int* __restrict__ Ct,
                                            const int32_t* __restrict__ rows, int r0, int r1,
                                            const uint8_t* __restrict__ codes, int stride, int fg0,
                                            const void* __restrict__ gqp, const void* __restrict__ hqp) {
    using T = ModeTraits<kMode>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int q = lane >> 2, sh = (lane & 3) * 8;
    const bool two_chunks = stride - fg0 >= 32;
    const bool v8 = two_chunks && (stride & 31) == 0;
    long long accG[kCells], accH[kCells];
    unsigned int accC[kCells];
#pragma unroll
    for (int cc = 0; cc < kCells; ++cc) {
        accG[cc] = 0;
        accH[cc] = 0;
        accC[cc] = 0u;
    }
    for (int s0 = r0; s0 < r1; s0 += T::sub) {
        const int s1 = min(r1, s0 + T::sub);
        int r_next = s0 + warp * 32 + lane < s1 ? rows[s0 + warp * 32 + lane] : -1;
        for (int base = s0 + warp * 32; base < s1; base += kWarps * 32) {
            const int r = r_next;
            const int k = base + lane;  // the row's position: its payload's index
            const int kn = base + kWarps * 32 + lane;
            r_next = kn < s1 ? rows[kn] : -1;
            if (r < 0) continue;
            unsigned int a0 = 0, a1 = 0, a2 = 0, a3 = 0;
            if constexpr (kMode == kHistExactVar) {
                const long long gv = static_cast<const long long*>(gqp)[k];
                const long long hv = static_cast<const long long*>(hqp)[k];
                a0 = static_cast<unsigned int>(gv) & ((1u << kLoBits) - 1u);
                a1 = static_cast<unsigned int>(static_cast<int>(gv >> kLoBits));
                a2 = static_cast<unsigned int>(hv) & ((1u << kLoBits) - 1u);
                a3 = static_cast<unsigned int>(static_cast<int>(hv >> kLoBits));
            } else if constexpr (kMode == kHistQ16Var) {
                const unsigned int p = static_cast<const unsigned int*>(gqp)[k];
                a0 = static_cast<unsigned int>(static_cast<int>(p) >> 16);
                a1 = p & 0xffffu;
            } else {  // kHistQ8Var
                const unsigned int p = static_cast<const unsigned short*>(gqp)[k];
                a0 = (1u << 20) | (p & 0xffu);
                a1 = p >> 8;
            }
            uint4 ca, cb;
            load_codes(codes + static_cast<size_t>(r) * stride + fg0, v8, two_chunks, ca, cb);
            unsigned int wd[8] = {ca.x, ca.y, ca.z, ca.w, cb.x, cb.y, cb.z, cb.w};
            rotate_words(wd, q);
            unsigned int Rw[8];
#pragma unroll
            for (int t = 0; t < 8; ++t) Rw[t] = __funnelshift_r(wd[t], wd[(t + 1) & 7], sh);
#pragma unroll
            for (int jj = 0; jj < 32; ++jj) {
                const int f = (jj + lane) & 31;
                const unsigned int code = (Rw[jj >> 2] >> ((jj & 3) * 8)) & 0xffu;
                const int cell = static_cast<int>(code) * 32 + f;
                if constexpr (kMode == kHistExactVar) {
                    atomicAdd(&P[cell], a0);
                    atomicAdd(&P[kPlane + cell], a1);
                    atomicAdd(&P[2 * kPlane + cell], a2);
                    atomicAdd(&P[3 * kPlane + cell], a3);
                    atomicAdd(&P[4 * kPlane + cell], 1u);
                } else if constexpr (kMode == kHistQ16Var) {
                    atomicAdd(&P[cell], a0);
                    atomicAdd(&P[kPlane + cell], a1);
                    atomicAdd(&P[2 * kPlane + cell], 1u);
                } else {
                    atomicAdd(&P[cell], a0);
                    atomicAdd(&P[kPlane + cell], a1);
                }
            }
        }
        __syncthreads();
        // fold the sub-chunk into 64-bit registers and clear the planes
#pragma unroll
        for (int cc = 0; cc < kCells; ++cc) {
            const int cell = threadIdx.x + cc * kThreads;
            if constexpr (kMode == kHistExactVar) {
                accG[cc] += static_cast<long long>(static_cast<int>(P[kPlane + cell])) * (1ll << kLoBits) + P[cell];
                accH[cc] +=
                    static_cast<long long>(static_cast<int>(P[3 * kPlane + cell])) * (1ll << kLoBits) + P[2 * kPlane + cell];
                accC[cc] += P[4 * kPlane + cell];
            } else if constexpr (kMode == kHistQ16Var) {
                accG[cc] += static_cast<int>(P[cell]);
                accH[cc] += P[kPlane + cell];
                accC[cc] += P[2 * kPlane + cell];
            } else {
                const unsigned int w1 = P[cell];
                const unsigned int n1 = w1 >> 20;
                accG[cc] += static_cast<long long>(w1 & 0xfffffu) - 128ll * static_cast<long long>(n1);
                accH[cc] += P[kPlane + cell];
                accC[cc] += n1;
            }
#pragma unroll
            for (int pl = 0; pl < T::planes; ++pl) P[pl * kPlane + cell] = 0u;
        }
        __syncthreads();
    }
    // totals over the (clear) planes: every cell of the padded layout has one owner
#pragma unroll
    for (int cc = 0; cc < kCells; ++cc) {
        const int cell = threadIdx.x + cc * kThreads;
        const int ti = (cell & 31) * kTotPitch + (cell >> 5);
        Gt[ti] = static_cast<unsigned long long>(accG[cc]);
        Ht[ti] = static_cast<unsigned long long>(accH[cc]);
        Ct[ti] = accC[cc];
    }
}

// One piece of a cluster's work: a CTA's rows of a (job, feature group) and where its sums go.
struct HistPiece {
    const int32_t* rows;
    const void* gq;
    const void* hq;
    unsigned long long hq1, hq2;  // fixed-point hessians of the two row classes
    size_t out0;                  // first cell of the group in the job's slot
    int c, r0, r1, fg0, nf, whole;
};

// A cell's totals summed over the cluster, and its hessian and count in the output's form.
template <bool kVar>
struct CellSum {
    unsigned long long g = 0, h = 0;
    unsigned int c = 0, c2 = 0;
};

// The end of a piece: every rank of a cluster of CS CTAs takes a share of the group's cells,
// adds it over the CTAs' shared totals (all loads before the first use) and writes it out.
// The CTAs may reuse their totals after the second barrier; its arrival comes before the
// global writes, so that nothing waits for those.
template <bool kVar, int CS>
__device__ __forceinline__ void flush_piece(const WaveCtx& X, const unsigned long long* Gt, const unsigned long long* Ht,
                                            const unsigned int* Ct, unsigned int rank, const HistPiece& piece) {
    const bool whole = piece.whole != 0;
    const unsigned long long hq1 = piece.hq1, hq2 = piece.hq2;
    const size_t out0 = piece.out0;
    constexpr int kIter = kPlane / CS / kThreads;  // cells a thread writes (8, 4 or 2)
    const int share = piece.nf * kBins / CS;
    const int i0 = static_cast<int>(rank) * share + static_cast<int>(threadIdx.x);
    const int i1 = static_cast<int>(rank + 1) * share;
    CellSum<kVar> v[kIter];
    if constexpr (CS > 1) cg::this_cluster().sync();
#pragma unroll
    for (int kk = 0; kk < CS; ++kk) {
        const unsigned long long* rG = CS > 1 ? cg::this_cluster().map_shared_rank(Gt, kk) : Gt;
        const unsigned long long* rH = CS > 1 ? cg::this_cluster().map_shared_rank(Ht, kk) : Ht;
        const unsigned int* rC = CS > 1 ? cg::this_cluster().map_shared_rank(Ct, kk) : Ct;
#pragma unroll
        for (int q = 0; q < kIter; ++q) {
            const int i = i0 + q * kThreads;
            if (i >= i1) continue;
            const int ti = i + (i >> 8);  // (feature i >> 8, bin i & 255) in the padded layout
            const unsigned int pc = rC[ti];
            v[q].g += rG[ti];
            if constexpr (kVar) {
                v[q].h += rH[ti];
                v[q].c += pc;
            } else {
                v[q].c += pc & 0xffffu;
                v[q].c2 += pc >> 16;
            }
        }
    }
    if constexpr (CS > 1) asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
#pragma unroll
    for (int q = 0; q < kIter; ++q) {
        const int i = i0 + q * kThreads;
        if (i >= i1) continue;
        unsigned long long h = v[q].h;
        unsigned int cn = v[q].c;
        if constexpr (!kVar) {
            h = static_cast<unsigned long long>(v[q].c) * hq1 + static_cast<unsigned long long>(v[q].c2) * hq2;
            cn += v[q].c2;
        }
        if (cn == 0u) continue;
        const size_t o = out0 + i;
        if (whole) {
            reinterpret_cast<unsigned long long*>(X.G)[o] = v[q].g;
            reinterpret_cast<unsigned long long*>(X.H)[o] = h;
            X.C[o] = static_cast<int>(cn);
        } else {
            atomicAdd(reinterpret_cast<unsigned long long*>(X.G) + o, v[q].g);
            atomicAdd(reinterpret_cast<unsigned long long*>(X.H) + o, h);
            atomicAdd(X.C + o, static_cast<int>(cn));
        }
    }
    if constexpr (CS > 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    else __syncthreads();
}

// One launch histograms every job (context, planned leaf's smaller child; or each
// context's root) of the wave.  The work, rows x feature groups summed over the jobs, is
// cut into one contiguous range per cluster; a cluster walks its range as pieces
// (job, feature group, row range), its CTAs split each piece's rows, and after a piece the
// cluster adds its CTAs' totals through distributed shared memory and writes them out:
// plain stores when the piece is the whole (job, feature group), 64-bit atomics when
// other clusters share it.  A job's slot is clear before the launch.
//
// The ranges: equal ones balance the rows but let a cluster straddle two (job, group)
// pairs, which costs it a second set-up, fold and flush.  Where there are at most 32 jobs
// and no more pairs than clusters, every pair gets clusters of its own in proportion to its
// rows, if the largest share then exceeds the equal one by less than that cost
// (kPieceRows rows a CTA).
//
// A child wave has a few hundred to a few thousand rows a CTA, so its launch is mostly fixed
// cost.  In cycles of one CTA at 100k x 32 the start took: plan 7,300 and piece set-up 5,500
// (chains of loads through the contexts and the node table: now one record a job, the
// contexts staged before the wait), flush 10,000 and the barrier and clearing after it 4,500
// (loads of one CTA's totals after another, global writes before the barrier: now all loads,
// the barrier, then the writes; nothing to clear).  Together with the pairs' own clusters:
// fits of 0.85M x 64 pairwise 92.2 -> 83.5 ms, 1.2M x 96 int8 97.0 -> 84.3 ms, 10M x 128
// 435 -> 416 ms.
//
// The plan and each piece's parameters are worked out by one warp and left in shared memory:
// 32 warps doing the same scalar work (64-bit divisions above all) took 8,000 cycles a piece.
//
// kPieceRows 0 (equal ranges only, nearly) / 500 / 1,500 / 5,000: 1.2M x 96 int8 73.8 / 64.5 / 64.8 /
// 64.7 ms, 0.85M x 64 pairwise 67.6 / 61.5 / 62 / 61.6, 20k x 16 35.8 / 32.8 / 32.3 / 31.4 (0.5 apart
// from run to run): anything but 0.  kMinCtaRows, below which a pair is not split further (a
// CTA's fold and flush cost more than its rows), 32 / 128 / 512: 64.4 / 64.8 / 64.4 and 31.5 / 32.3 /
// 32.4 ms, within the noise.
constexpr int kPieceRows = 1500;
constexpr int kMinCtaRows = 128;
constexpr int kWarpJobs = 32;

template <int kMode>
__global__ void __launch_bounds__(kThreads, 1)
    wave_hist_kernel(const WaveCtx* __restrict__ ctxs, int n_ctx, int src, unsigned long long* rows_counter) {
    using T = ModeTraits<kMode>;
    using Lay = SmemLayout<kMode>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned int* P = reinterpret_cast<unsigned int*>(smem_raw);  // working planes
    unsigned long long* Gt = reinterpret_cast<unsigned long long*>(smem_raw + Lay::tot_off);
    unsigned long long* Ht = Gt + kTot;  // per-row hessian modes only
    unsigned int* Ct = reinterpret_cast<unsigned int*>(Gt + (T::var ? 2 : 1) * kTot);
    unsigned long long* s_wstart = reinterpret_cast<unsigned long long*>(smem_raw + Lay::plan_off);
    // TMA staging (constant-hessian modes): slots over Gt from its first 128-byte boundary,
    // two mbarriers per warp, their parities
    __shared__ __align__(8) unsigned long long s_bars[2 * kWarps];
    __shared__ WaveCtx s_ctx;  // the first context's constants
    unsigned char* stage = smem_raw + Lay::tot_off;
    stage += (128u - (smem_u32(stage) & 127u)) & 127u;
    unsigned int phase = 0u;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // What does not depend on the previous kernel first, so that it overlaps its tail: the
    // private state, the barriers, and the context's constants (written by a host copy before
    // the fit's first tree), its TMA descriptor included.
    {
        uint4* z = reinterpret_cast<uint4*>(smem_raw);
        for (int k = threadIdx.x; k < static_cast<int>(Lay::work / 16); k += blockDim.x) z[k] = make_uint4(0, 0, 0, 0);
    }
    stage_ctx(s_ctx, ctxs);
    if (!T::var && lane == 0) {
        mbar_init(smem_u32(&s_bars[2 * warp]));
        mbar_init(smem_u32(&s_bars[2 * warp + 1]));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (!T::var && lane < 8)
        for (int c = 0; c < n_ctx; ++c)
            asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(&ctxs[c].codes_map) : "memory");
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    auto ctx_of = [&](int c) -> const WaveCtx& { return c == 0 ? s_ctx : ctxs[c]; };

    // ---- work plan (the same in every CTA) ----
    __shared__ int s_cpref[kMaxWaveCtx + 1];
    __shared__ unsigned long long s_red[kWarps], s_rsum[kWarps];
    __shared__ HistPiece s_piece;
    __shared__ int s_more, s_aligned;
    cg::cluster_group cluster = cg::this_cluster();
    const int csize = static_cast<int>(cluster.dim_blocks().y);  // CTAs per cluster: 1, 2 or 4
    const int cl = static_cast<int>(blockIdx.y) / csize;
    const int n_cl = static_cast<int>(gridDim.y) / csize;
    const unsigned int rank = csize > 1 ? cluster.block_rank() : 0u;
    // warp 0 only: the cluster's own pair (aligned), and how far its rows are handed out
    bool aligned = false;
    int a_job = -1, a_fg = 0, a_rows = 0, a_row = 0, a_end = 0;
    if (warp == 0) {
        // with one context the lane's job is read along with the number of jobs
        int early = 0;
        if (n_ctx == 1) early = job_count(s_ctx, src, lane);
        int all = 0;
        for (int c0 = 0; c0 < n_ctx; c0 += 32) {
            const int c = c0 + lane;
            int v = 0;
            if (c < n_ctx) v = src == 0 ? (ctx_of(c).ctl->active ? 1 : 0) : ctx_of(c).ctl->n_exp;
            int incl = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            if (c < n_ctx) s_cpref[c] = all + incl - v;
            all += __shfl_sync(0xffffffffu, incl, 31);
        }
        const int nj = min(all, kMaxWaveJobs);
        if (lane == 0) {
            s_cpref[n_ctx] = nj;
            s_aligned = 0;
        }
        __syncwarp();
        if (nj <= kWarpJobs) {
            // a lane per job: the work prefix, and the clusters of each of the job's pairs
            int count = 0, groups = 0;
            if (lane < nj) {
                int c = 0;
                while (c + 1 < n_ctx && s_cpref[c + 1] <= lane) ++c;
                count = n_ctx == 1 ? early : job_count(ctx_of(c), src, lane - s_cpref[c]);
                groups = (ctx_of(c).gp.n_features + kFG - 1) / kFG;
            }
            const unsigned long long w = static_cast<unsigned long long>(count) * groups;
            unsigned long long incl = w;
            unsigned int rows = static_cast<unsigned int>(count);
            int pairs = groups;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
                pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
            }
            const unsigned long long w_all = __shfl_sync(0xffffffffu, incl, 31);
            if (lane < nj) s_wstart[lane] = incl - w;
            if (lane == 0) s_wstart[nj] = w_all;
            if (rows_counter != nullptr && blockIdx.y == 0) {
                unsigned long long r = rows;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
                if (lane == 0) atomicAdd(rows_counter, r);
            }
            if (pairs <= n_cl && w_all > 0) {
                // one cluster a pair, the others in proportion to the rows (rounded down), then
                // what is left one by one to the largest share
                const float spare = static_cast<float>(n_cl - pairs) / static_cast<float>(w_all) * 0.9999f;
                const int cap = max(1, (count + kMinCtaRows * csize - 1) / (kMinCtaRows * csize));
                int per = min(1 + static_cast<int>(spare * static_cast<float>(count)), cap);
                int used = groups * per;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) used += __shfl_xor_sync(0xffffffffu, used, o);
                for (int it = 0; it < 8; ++it) {
                    const bool can = groups > 0 && per < cap && groups <= n_cl - used;
                    // positive floats order like their bits; 0: no job can take another cluster
                    const unsigned share = can ? __float_as_uint(__fdividef(static_cast<float>(count), static_cast<float>(per))) : 0u;
                    const unsigned top = __reduce_max_sync(0xffffffffu, share);
                    if (top == 0u) break;
                    const int who = __ffs(__ballot_sync(0xffffffffu, share == top)) - 1;
                    if (lane == who) ++per;
                    used += __shfl_sync(0xffffffffu, groups, who);
                }
                float most = groups > 0 ? static_cast<float>(count) / static_cast<float>(per) : 0.f;
                int cs = groups * per;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
                    const int t = __shfl_up_sync(0xffffffffu, cs, o);
                    if (lane >= o) cs += t;
                }
                if (most <= static_cast<float>(w_all) / static_cast<float>(n_cl) + static_cast<float>(kPieceRows * csize)) {
                    // this cluster's pair: the job whose clusters hold it, the pair's rows in
                    // per equal parts (the first ones a row longer)
                    aligned = true;
                    const unsigned mine = __ballot_sync(0xffffffffu, cl >= cs - groups * per && cl < cs);
                    const int src_lane = mine ? __ffs(mine) - 1 : 0;
                    a_job = mine ? src_lane : -1;
                    const int q = cl - __shfl_sync(0xffffffffu, cs - groups * per, src_lane);
                    const int jper = __shfl_sync(0xffffffffu, per, src_lane), R = __shfl_sync(0xffffffffu, count, src_lane);
                    a_fg = q / jper;
                    const int k = q - a_fg * jper, part = R / jper, longer = R - part * jper;
                    a_rows = R;
                    a_row = part * k + min(k, longer);
                    a_end = a_row + part + (k < longer ? 1 : 0);
                    if (lane == 0) s_aligned = 1;
                }
            }
        }
    }
    __syncthreads();
    const int n_jobs = s_cpref[n_ctx];
    if (n_jobs > kWarpJobs) {
        // work of each job (rows x feature groups), exclusive prefix over a contiguous run
        // of jobs per thread
        const int per = (n_jobs + kThreads - 1) / kThreads;
        const int j0 = min(n_jobs, static_cast<int>(threadIdx.x) * per), j1 = min(n_jobs, j0 + per);
        unsigned long long local = 0, lrows = 0;
        for (int j = j0; j < j1; ++j) {
            int c = 0;
            while (c + 1 < n_ctx && s_cpref[c + 1] <= j) ++c;
            const int count = job_count(ctx_of(c), src, j - s_cpref[c]);
            const unsigned long long w =
                static_cast<unsigned long long>(count) * ((ctx_of(c).gp.n_features + kFG - 1) / kFG);
            s_wstart[j] = w;
            local += w;
            lrows += static_cast<unsigned long long>(count);
        }
        unsigned long long incl = local, rs = lrows;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
            rs += __shfl_xor_sync(0xffffffffu, rs, o);
        }
        if (lane == 31) s_red[warp] = incl;
        if (lane == 0) s_rsum[warp] = rs;
        __syncthreads();
        unsigned long long wbase = 0, all = 0, rows_all = 0;
        for (int k = 0; k < kWarps; ++k) {
            if (k < warp) wbase += s_red[k];
            all += s_red[k];
            rows_all += s_rsum[k];
        }
        unsigned long long run = wbase + incl - local;
        for (int j = j0; j < j1; ++j) {
            const unsigned long long w = s_wstart[j];
            s_wstart[j] = run;
            run += w;
        }
        if (threadIdx.x == 0) {
            s_wstart[n_jobs] = all;
            if (rows_counter != nullptr && blockIdx.y == 0) atomicAdd(rows_counter, rows_all);
        }
        __syncthreads();
    }
    unsigned long long w = 0, w_end = 0;  // warp 0, without pairs of their own: the range's work
    if (warp == 0 && !s_aligned) {
        const unsigned long long w_all = s_wstart[n_jobs];
        w = w_all * static_cast<unsigned long long>(cl) / static_cast<unsigned long long>(n_cl);
        w_end = w_all * static_cast<unsigned long long>(cl + 1) / static_cast<unsigned long long>(n_cl);
    }
    const int max_piece = kMaxShareRows * csize;
    while (true) {
        if (warp == 0) {
            // the next piece: job, feature group and rows
            int j = -1, fg = 0, R = 0, piece0 = 0, piece1 = 0;
            if (aligned) {
                if (a_row < a_end && a_job >= 0) {
                    j = a_job;
                    fg = a_fg;
                    R = a_rows;
                    piece0 = a_row;
                    piece1 = min(a_end, a_row + max_piece);
                    a_row = piece1;
                }
            } else if (w < w_end) {
                // the job holding w: the last j with s_wstart[j] <= w (a non-empty job)
                int lo = 0, hi = n_jobs - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (s_wstart[mid] <= w) lo = mid;
                    else hi = mid - 1;
                }
                j = lo;
                int c = 0;
                while (c + 1 < n_ctx && s_cpref[c + 1] <= j) ++c;
                R = job_count(ctx_of(c), src, src == 0 ? 0 : j - s_cpref[c]);
                const unsigned long long off = w - s_wstart[j];
                fg = static_cast<int>(off / static_cast<unsigned long long>(R));
                piece0 = static_cast<int>(off - static_cast<unsigned long long>(fg) * R);
                const unsigned long long len =
                    min(min(static_cast<unsigned long long>(R - piece0), w_end - w), static_cast<unsigned long long>(max_piece));
                piece1 = piece0 + static_cast<int>(len);
                w += len;
            }
            if (lane == 0) s_more = j >= 0;
            if (j >= 0) {
                int c = 0;
                while (c + 1 < n_ctx && s_cpref[c + 1] <= j) ++c;
                const WaveCtx& X = ctx_of(c);
                if (lane == 0) {
                    const JobRows jr = job_rows(X, src, src == 0 ? 0 : j - s_cpref[c]);
                    const int q = (piece1 - piece0 + csize - 1) / csize;
                    HistPiece p;
                    p.rows = jr.rows;
                    p.gq = jr.gq;
                    p.hq = jr.hq;
                    p.c = c;
                    p.r0 = min(piece1, piece0 + static_cast<int>(rank) * q);
                    p.r1 = min(piece1, p.r0 + q);
                    p.fg0 = fg * kFG;
                    p.nf = min(kFG, X.gp.n_features - p.fg0);
                    p.whole = piece0 == 0 && piece1 == R;
                    p.out0 = (static_cast<size_t>(jr.slot) * static_cast<size_t>(X.gp.n_features) + p.fg0) * kBins;
                    p.hq1 = p.hq2 = 0ull;
                    if (!T::var) {
                        const double hscale = X.st->hscale;
                        p.hq1 = static_cast<unsigned long long>(__double2ll_rn(1.0 * hscale));
                        p.hq2 = static_cast<unsigned long long>(__double2ll_rn(1.0 * X.goss_scale * hscale));
                    }
                    s_piece = p;
                }
            }
        }
        __syncthreads();
        if (!s_more) break;
        const WaveCtx& X = ctx_of(s_piece.c);
        if constexpr (T::var)
            accumulate_var<kMode>(P, Gt, Ht, Ct, s_piece.rows, s_piece.r0, s_piece.r1, X.codes, X.gp.stride, s_piece.fg0,
                                  s_piece.gq, s_piece.hq);
        else if (X.codes_map_ok && (reinterpret_cast<uintptr_t>(&ctxs[s_piece.c].codes_map) & 63u) == 0)  // TMA: 64 B
            phase = accumulate_const_tma<kMode>(P, Gt, Ct, stage, s_bars, phase, s_piece.rows, s_piece.r0, s_piece.r1,
                                                &ctxs[s_piece.c].codes_map, s_piece.fg0, s_piece.gq, &X.ctl->error);
        else
            accumulate_const<kMode>(P, Gt, Ct, s_piece.rows, s_piece.r0, s_piece.r1, X.codes, X.gp.stride, s_piece.fg0,
                                    s_piece.gq);
        __syncthreads();
        if (csize == 1) flush_piece<T::var, 1>(X, Gt, Ht, Ct, rank, s_piece);
        else if (csize == 2) flush_piece<T::var, 2>(X, Gt, Ht, Ct, rank, s_piece);
        else flush_piece<T::var, 4>(X, Gt, Ht, Ct, rank, s_piece);
        if (T::var) {  // the totals lie over the planes: clear for a next piece (rare: most take one)
            if (warp == 0 && lane == 0) s_more = aligned ? a_row < a_end : w < w_end;
            __syncthreads();
            if (!s_more) break;
            uint4* z = reinterpret_cast<uint4*>(smem_raw);
            for (int k = threadIdx.x; k < static_cast<int>(Lay::region / 16); k += kThreads) z[k] = make_uint4(0, 0, 0, 0);
            __syncthreads();
        }
    }
}

// ---- partition ----------------------------------------------------------------------
constexpr int kPartThreads = 256;
constexpr int kPartWarps = kPartThreads / 32;
constexpr int kPartPer = kPartTile / kPartThreads;

// A row's g payload (element i of the payload array), widened to 64 bits, and back.
__device__ __forceinline__ long long load_payload(const WaveCtx& X, long long i) {
    if (X.pay_bytes == 8) return static_cast<const long long*>(X.gq)[i];
    if (X.pay_bytes == 4) return static_cast<const int*>(X.gq)[i];
    return static_cast<const short*>(X.gq)[i];
}
__device__ __forceinline__ void store_payload(const WaveCtx& X, long long i, long long v) {
    if (X.pay_bytes == 8) static_cast<long long*>(X.gq)[i] = v;
    else if (X.pay_bytes == 4) static_cast<int*>(X.gq)[i] = static_cast<int>(v);
    else static_cast<short*>(X.gq)[i] = static_cast<short>(v);
}

// One launch moves the rows of every planned leaf into its children.  A tile of 2048 rows
// ranks its rows by side with ballots, reserves its places in both children with one 64-bit
// atomic add on the leaf's cursor (left rows in the low word, right rows in the high word)
// and writes them: left rows upward from the leaf's start, right rows in blocks downward
// from its end, so no tile needs the leaf's left total.  The tile whose reservation
// completes the leaf knows that total and writes the children's ranges.
//
// Inside a tile the row order is kept, between tiles it depends on which reserves first.
// Every use of a row list is an exact integer sum, so no result depends on the order, and a
// child's list still runs over ascending row ids tile by tile, which is what the gathers of
// codes need.  The reference's stable order took two launches (count, then scatter from the
// tile prefixes): both are bound by their chain of dependent loads, and the second read the
// rows and codes again.
// kPair: some context searches PAIR splits, so the children's gradient energies (sums of g^2,
// exact in fixed point) are made on the way.
template <bool kPair>
__global__ void __launch_bounds__(kPartThreads)
    wave_part_kernel(const WaveCtx* __restrict__ ctxs, int n_ctx) {
    __shared__ WaveCtx s_ctx;  // the first context's constants
    __shared__ int s_pref[kMaxWaveCtx + 1];
    __shared__ int wc[kPartWarps];
    __shared__ unsigned long long s_old, s_en[2];
    stage_ctx(s_ctx, ctxs);
    __syncthreads();
    pdl_wait();
    pdl_trigger();
    auto ctx_of = [&](int c) -> const WaveCtx& { return c == 0 ? s_ctx : ctxs[c]; };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    if (warp == 0) {
        int all = 0;
        for (int c0 = 0; c0 < n_ctx; c0 += 32) {
            const int c = c0 + lane;
            const int v = c < n_ctx ? ctx_of(c).ctl->tiles_total : 0;
            int incl = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            if (c < n_ctx) s_pref[c] = all + incl - v;
            all += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) s_pref[n_ctx] = all;
    }
    __syncthreads();
    const int total = s_pref[n_ctx];
    // Clear the histogram slots of this wave's children (2 per expansion, consecutive): the
    // smaller child's is accumulated into by the histogram launch.  First, so that the stores
    // drain while the tiles wait for their loads.
    for (int c = 0; c < n_ctx; ++c) {
        const WaveCtx& X = ctx_of(c);
        const int ns = 2 * X.ctl->n_exp;
        if (ns == 0) continue;
        const size_t elems = static_cast<size_t>(X.gp.n_features) * kBins;
        const size_t first = static_cast<size_t>(X.ctl->slot0) * elems;
        const size_t n8 = static_cast<size_t>(ns) * elems;  // int64 elements of G and H
        uint4* g4 = reinterpret_cast<uint4*>(X.G + first);
        uint4* h4 = reinterpret_cast<uint4*>(X.H + first);
        uint4* c4 = reinterpret_cast<uint4*>(X.C + first);
        const size_t n16_8 = n8 / 2, n16_4 = n8 / 4;  // elems is a multiple of 256
        for (size_t k = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; k < n16_8;
             k += static_cast<size_t>(gridDim.x) * blockDim.x) {
            g4[k] = make_uint4(0, 0, 0, 0);
            h4[k] = make_uint4(0, 0, 0, 0);
            if (k < n16_4) c4[k] = make_uint4(0, 0, 0, 0);
        }
    }
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
        int c = 0;
        while (c + 1 < n_ctx && s_pref[c + 1] <= t) ++c;
        const WaveCtx& X = ctx_of(c);
        WaveCtl* ctl = X.ctl;
        // the expansion of tile t: the last one that starts at or before it (every warp counts
        // the starts, 32 at a time)
        const int lt = t - s_pref[c], n_exp = ctl->n_exp;
        int e = -1;
        for (int e0 = 0; e0 < n_exp; e0 += 32) {
            const int first = ctl->exp_tile0[e0 + lane];  // the array is longer than its use
            e += __popc(__ballot_sync(0xffffffffu, e0 + lane < n_exp && first <= lt));
        }
        const WaveExp S = ctl->exp[e];
        const int L = S.leaf, count = S.count;
        const int32_t* in = (S.buf ? X.rows1 : X.rows0) + S.start;
        int32_t* out = (S.buf ? X.rows0 : X.rows1) + S.start;
        const int base = (lt - ctl->exp_tile0[e]) * kPartTile, end = min(base + kPartTile, count);
        // a warp takes 256 consecutive rows, 32 at a time; the rows' payloads move with them
        // (same positions in the other buffer), so their loads go out with the row ids'
        const long long from0 = static_cast<long long>(S.buf) * X.pay_pitch + S.start;
        const long long to0 = static_cast<long long>(1 - S.buf) * X.pay_pitch + S.start;
        const int k0 = base + warp * (32 * kPartPer) + lane;
        int32_t row[kPartPer];
        long long pg[kPartPer], ph[kPartPer];
#pragma unroll
        for (int i = 0; i < kPartPer; ++i) row[i] = k0 + 32 * i < end ? in[k0 + 32 * i] : -1;
#pragma unroll
        for (int i = 0; i < kPartPer; ++i) {
            const int kk = k0 + 32 * i;
            pg[i] = kk < end ? load_payload(X, from0 + kk) : 0;
            ph[i] = kk < end && X.hq != nullptr ? static_cast<const long long*>(X.hq)[from0 + kk] : 0;
        }
        unsigned int b[kPartPer], b2[kPartPer];
        const uint8_t* col = X.codes_col + static_cast<size_t>(S.feature) * X.col_pitch;
        const uint8_t* col2 = S.type == 1 ? X.codes_col + static_cast<size_t>(S.feature2) * X.col_pitch : col;
#pragma unroll
        for (int i = 0; i < kPartPer; ++i) {
            b[i] = row[i] >= 0 ? col[row[i]] : 0u;
            b2[i] = row[i] >= 0 && S.type == 1 ? col2[row[i]] : 0u;
        }
        // PAIR: the rows' g^2 as the tree sees them (GOSS-scaled), in fixed point
        unsigned long long en[kPair ? kPartPer : 1];
        if (kPair && X.pair_on) {
            const double scale = ldexp(1.0, energy_shift(X.st));
#pragma unroll
            for (int i = 0; i < (kPair ? kPartPer : 0); ++i) {
                double gv = row[i] >= 0 ? X.g[row[i]] : 0.0;
                if (row[i] >= 0 && X.goss_flag != nullptr && X.goss_flag[row[i]] == 2) gv *= X.goss_scale;
                en[i] = static_cast<unsigned long long>(__double2ll_rn(gv * gv * scale));
            }
            if (threadIdx.x < 2) s_en[threadIdx.x] = 0ull;
        }
        unsigned bal[kPartPer];
        int excl[kPartPer];  // left rows of the warp's earlier 32s, then of the tile's earlier rows
        int mine = 0;
#pragma unroll
        for (int i = 0; i < kPartPer; ++i) {
            const bool l =
                row[i] >= 0 && goes_left(S.type, S.cat, S.threshold, S.missing_left, b[i], b2[i], X.gp.n_bins);
            bal[i] = __ballot_sync(0xffffffffu, l);
            excl[i] = mine;
            mine += __popc(bal[i]);
        }
        if (lane == 0) wc[warp] = mine;
        __syncthreads();
        if (kPair && X.pair_on) {
            unsigned long long el = 0, er = 0;
#pragma unroll
            for (int i = 0; i < (kPair ? kPartPer : 0); ++i) {
                if ((bal[i] >> lane) & 1u) el += en[i];
                else er += en[i];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                el += __shfl_xor_sync(0xffffffffu, el, o);
                er += __shfl_xor_sync(0xffffffffu, er, o);
            }
            if (lane == 0) {
                atomicAdd(&s_en[0], el);
                atomicAdd(&s_en[1], er);
            }
        }
        int run = 0;  // the tile's left rows
        int before = 0;
#pragma unroll
        for (int w = 0; w < kPartWarps; ++w) {
            const int cw = wc[w];
            if (w < warp) before += cw;
            run += cw;
        }
        const int n_right = end - base - run;
        if (threadIdx.x == 0) {
            const unsigned long long old =
                atomicAdd(&ctl->part_cur[e],
                          (static_cast<unsigned long long>(n_right) << 32) | static_cast<unsigned int>(run));
            s_old = old;
            const int l0 = static_cast<int>(old & 0xffffffffu), r0 = static_cast<int>(old >> 32);
            if (l0 + r0 + (end - base) == count) {
                DevNode& A = X.spec[2 * L];
                DevNode& B = X.spec[2 * L + 1];
                const int nl = l0 + run, nr = count - nl, slot = S.child_slot;
                A.start = S.start;
                A.count = nl;
                B.start = S.start + nl;
                B.count = nr;
                const bool ls = nl <= nr;  // the left child is the smaller one (cpp/src/tree.cpp:423)
                ctl->job[e] = WaveJob{ls ? S.start : S.start + nl, ls ? nl : nr, 1 - S.buf, ls ? slot : slot + 1};
                const bool deep = S.depth + 1 < X.gp.max_depth;
                const int need = 2 * X.gp.min_samples_leaf;
                ctl->child[2 * e] = WaveChild{2 * L, slot, S.slot, slot + 1, !ls, deep && nl >= need, {0, 0}};
                ctl->child[2 * e + 1] = WaveChild{2 * L + 1, slot + 1, S.slot, slot, ls, deep && nr >= need, {0, 0}};
            }
        }
        __syncthreads();
        if (kPair && X.pair_on && threadIdx.x < 2) atomicAdd(&X.energy[2 * L + threadIdx.x], s_en[threadIdx.x]);
        const int left0 = static_cast<int>(s_old & 0xffffffffu);
        const int right0 = count - static_cast<int>(s_old >> 32) - n_right;
#pragma unroll
        for (int i = 0; i < kPartPer; ++i) {
            if (row[i] < 0) continue;
            const int kk = k0 + 32 * i;
            const int lrank = before + excl[i] + __popc(bal[i] & lt_mask);
            const bool l = (bal[i] >> lane) & 1u;
            const int dst = l ? left0 + lrank : right0 + (kk - base - lrank);
            out[dst] = row[i];
            store_payload(X, to0 + dst, pg[i]);
            if (X.hq != nullptr) static_cast<long long*>(X.hq)[to0 + dst] = ph[i];
        }
        __syncthreads();  // wc and s_old reuse
    }
}

// ---- per-tree set-up ------------------------------------------------------------------
// The root node and the control of a new tree (one thread).
__device__ __forceinline__ void init_tree(DevNode* nodes, DevSplit* splits, DevTreeState* st, WaveCtl* ctl, int count) {
    DevNode r{};
    r.start = 0;
    r.count = count;
    r.buf = 0;
    r.depth = 0;
    r.is_leaf = 1;
    r.feature = -1;
    r.threshold = -1;
    r.missing_left = 1;
    r.left = r.right = r.parent = -1;
    r.slot = 0;
    nodes[0] = r;
    splits[0].valid = 0;
    st->n_nodes = 1;
    st->done = 0;
    st->parent = -1;
    st->small_node = st->large_node = -1;
    st->n_sample = count;
    ctl->splits_done = 0;
    ctl->n_exp = 0;
    ctl->exp_counter = 0;
    ctl->tiles_total = 0;
    ctl->active = 1;
    ctl->slot0 = 1;
    ctl->waves = 0;
    ctl->pair_used = 0;
    ctl->expanded[0] = 0;
}

__device__ int shift_for(double max_abs, int count) {
    if (!(max_abs > 0.0) || count <= 0) return 0;
    int clog = 0;
    while ((1ll << clog) < static_cast<long long>(count)) ++clog;
    const int e = ilogb(max_abs);
    int s = min(61 - (e + 1) - clog, 36 - e);
    return max(-1000, min(1000, s));
}

// Exact modes: power-of-two shifts (no sum over the sample can reach 2^62, no row's value
// 2^37).  Quantised modes: the largest |g| (and h) of the sample maps to the largest
// code; constant-hessian modes keep the exact hessian shift (H is rebuilt from counts).
__device__ __forceinline__ void set_scales(DevTreeState* st, const AllScale* __restrict__ all, int mode) {
    if (all) {
        st->max_abs_g_bits = all->maxg_bits;
        st->max_h_bits = all->maxh_bits;
    }
    const double mg = __longlong_as_double(static_cast<long long>(st->max_abs_g_bits));
    const double mh = __longlong_as_double(static_cast<long long>(st->max_h_bits));
    const bool var = mode & 1;
    const int qbits = mode >= kHistQ8Const ? 8 : mode >= kHistQ16Const ? 16 : 0;
    if (qbits == 0) {
        st->gshift = shift_for(mg, st->n_sample);
        st->gscale = ldexp(1.0, st->gshift);
        st->inv_gscale = ldexp(1.0, -st->gshift);
    } else {
        const double gmax = qbits == 8 ? 127.0 : 32767.0;
        st->gshift = 0;
        st->gscale = mg > 0.0 ? gmax / mg : 1.0;
        st->inv_gscale = 1.0 / st->gscale;
    }
    if (qbits == 0 || !var) {
        st->hshift = shift_for(mh, st->n_sample);
        st->hscale = ldexp(1.0, st->hshift);
        st->inv_hscale = ldexp(1.0, -st->hshift);
    } else {
        const double hmax = qbits == 8 ? 255.0 : 65535.0;
        st->hshift = 0;
        st->hscale = mh > 0.0 ? hmax / mh : 1.0;
        st->inv_hscale = 1.0 / st->hscale;
    }
}

__global__ void wave_scales_kernel(DevTreeState* st, const AllScale* __restrict__ all, int mode) {
    set_scales(st, all, mode);
}

// Everything between the gradients (and the GOSS sample) and the payloads of a new tree, in one
// launch: the all-row scales, the root, the control and the histogram scales by one thread; the
// root's histogram slot, the segment sums and the root's energy cleared and, without GOSS,
// the row list written by the others.  (Nine launches of a few microseconds each before.)
__global__ void __launch_bounds__(256) wave_begin_kernel(WaveBegin a) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        finalize_all_scale(a.all, a.n);
        init_tree(a.nodes, a.splits, a.st, a.ctl, a.sampled ? a.st->n_sample : a.n);
        set_scales(a.st, a.sampled ? nullptr : a.all, a.mode);
        if (a.energy != nullptr) *a.energy = 0ull;
    }
    const size_t at = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x, step = static_cast<size_t>(gridDim.x) * blockDim.x;
    const uint4 zero = make_uint4(0, 0, 0, 0);
    for (size_t k = at; k < a.slot_elems / 2; k += step) {  // slot_elems is a multiple of 256
        reinterpret_cast<uint4*>(a.G)[k] = zero;
        reinterpret_cast<uint4*>(a.H)[k] = zero;
        if (k < a.slot_elems / 4) reinterpret_cast<uint4*>(a.C)[k] = zero;
    }
    for (size_t k = at; k < a.seg_words; k += step) a.seg_sums[k] = 0ull;
    if (!a.sampled)
        for (size_t k = at; k < static_cast<size_t>(a.n); k += step) a.rows0[k] = static_cast<int32_t>(k);
}

// SplitMix64 output function (Steele, Lea and Flood, OOPSLA 2014): the stream of uniform
// numbers of the stochastic rounding, a function of (row, tree, seed) only.
__device__ __forceinline__ unsigned long long splitmix64(unsigned long long z) {
    z += 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}

__device__ __forceinline__ double uniform01(unsigned long long seed, int r, unsigned salt) {
    const unsigned long long z = splitmix64(seed ^ (static_cast<unsigned long long>(r) << 20) ^
                                            (static_cast<unsigned long long>(salt) << 52));
    return static_cast<double>(z >> 11) * (1.0 / 9007199254740992.0);  // 53 bits -> [0, 1)
}

// floor(x + u), u uniform in [0, 1): unbiased stochastic rounding, clamped to [lo, hi].
__device__ __forceinline__ int sround(double x, double u, int lo, int hi) {
    return max(lo, min(hi, static_cast<int>(floor(x + u))));
}

template <int kMode>
__global__ void wave_quantize_kernel(const int32_t* __restrict__ rows, const double* __restrict__ g,
                                     const double* __restrict__ h, const uint8_t* __restrict__ goss_flag,
                                     double goss_scale, const DevTreeState* __restrict__ st,
                                     unsigned long long seed, bool per_tree, void* __restrict__ gq,
                                     void* __restrict__ hq, unsigned long long* __restrict__ energy) {
    if (per_tree) seed = splitmix64(seed + static_cast<unsigned long long>(st->tree));
    const int count = st->n_sample;
    const double escale = energy != nullptr ? ldexp(1.0, energy_shift(st)) : 0.0;
    unsigned long long en = 0;
    const double gscale = st->gscale, hscale = st->hscale;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
        const int r = rows[k];
        double gv = g[r];
        double hv = h ? h[r] : 1.0;
        const bool sc = goss_flag != nullptr && goss_flag[r] == 2;
        if (sc) {
            gv *= goss_scale;
            hv *= goss_scale;
        }
        if (energy != nullptr) en += static_cast<unsigned long long>(__double2ll_rn(gv * gv * escale));
        if constexpr (kMode == kHistExactConst) {
            const long long v = __double2ll_rn(gv * gscale);
            static_cast<long long*>(gq)[k] = static_cast<long long>((static_cast<unsigned long long>(v) << 1) | (sc ? 1ull : 0ull));
        } else if constexpr (kMode == kHistExactVar) {
            static_cast<long long*>(gq)[k] = __double2ll_rn(gv * gscale);
            static_cast<long long*>(hq)[k] = __double2ll_rn(hv * hscale);
        } else if constexpr (kMode == kHistQ16Const) {
            const int qv = sround(gv * gscale, uniform01(seed, r, 0), -32767, 32767);
            static_cast<int*>(gq)[k] = static_cast<int>((static_cast<unsigned int>(qv) << 1) | (sc ? 1u : 0u));
        } else if constexpr (kMode == kHistQ16Var) {
            const int qg = sround(gv * gscale, uniform01(seed, r, 0), -32767, 32767);
            const int qh = sround(hv * hscale, uniform01(seed, r, 1), 0, 65535);
            static_cast<unsigned int*>(gq)[k] = (static_cast<unsigned int>(qg) << 16) | static_cast<unsigned int>(qh);
        } else if constexpr (kMode == kHistQ8Const) {
            const int qv = sround(gv * gscale, uniform01(seed, r, 0), -127, 127);
            static_cast<short*>(gq)[k] = static_cast<short>((qv * 2) | (sc ? 1 : 0));
        } else {
            const int qg = sround(gv * gscale, uniform01(seed, r, 0), -127, 127);
            const int qh = sround(hv * hscale, uniform01(seed, r, 1), 0, 255);
            static_cast<unsigned short*>(gq)[k] = static_cast<unsigned short>((qg + 128) | (qh << 8));
        }
    }
    if (energy != nullptr) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) en += __shfl_xor_sync(0xffffffffu, en, o);
        if ((threadIdx.x & 31) == 0 && en != 0ull) atomicAdd(energy, en);
    }
}

__global__ void rows_max_kernel(const int32_t* __restrict__ rows, int n_rows, const double* __restrict__ g,
                                const double* __restrict__ h, AllScale* __restrict__ sc) {
    double mg = 0.0, mh = 0.0;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n_rows; k += gridDim.x * blockDim.x) {
        const int r = rows[k];
        mg = fmax(mg, fabs(g[r]));
        mh = fmax(mh, h ? fabs(h[r]) : 1.0);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mg = fmax(mg, __shfl_xor_sync(0xffffffffu, mg, o));
        mh = fmax(mh, __shfl_xor_sync(0xffffffffu, mh, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&sc->maxg_bits, static_cast<unsigned long long>(__double_as_longlong(mg)));
        atomicMax(&sc->maxh_bits, static_cast<unsigned long long>(__double_as_longlong(mh)));
    }
}

template <typename K>
void set_smem(K kern, size_t bytes) {
    check(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)),
          "wave hist smem attr");
}

// The shared-memory opt-in of each histogram instantiation, set once per device.
template <int kMode>
void ensure_smem() {
    static std::atomic<bool> done[64] = {};
    int dev = 0;
    check(cudaGetDevice(&dev), "cudaGetDevice");
    if (dev >= 0 && dev < 64 && done[dev]) return;
    set_smem(wave_hist_kernel<kMode>, SmemLayout<kMode>::bytes);
    if (dev >= 0 && dev < 64) done[dev] = true;
}

template <int kMode>
void hist_launch(const WaveCtx* ctxs, int n_ctx, int src, HistTune tune, unsigned long long* rows_counter,
                 cudaStream_t s) {
    auto kern = wave_hist_kernel<kMode>;
    ensure_smem<kMode>();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1, tune.clusters * tune.cluster);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = SmemLayout<kMode>::bytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = tune.cluster;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = src == 0 && n_ctx > 1 ? 1 : 2;  // (the roots follow several streams' kernels)
    check(cudaLaunchKernelEx(&cfg, kern, ctxs, n_ctx, src, rows_counter), "wave_hist launch");
}

template <int kMode>
void quantize_launch(const int32_t* rows, const double* g, const double* h, const uint8_t* flag, double gs,
                     const DevTreeState* st, unsigned long long seed, bool per_tree, void* gq, void* hq,
                     unsigned long long* energy, int blocks, cudaStream_t s) {
    wave_quantize_kernel<kMode><<<blocks, 256, 0, s>>>(rows, g, h, flag, gs, st, seed, per_tree, gq, hq, energy);
}

}  // namespace

int wave_hist_clusters(int cluster) {
    static std::atomic<int> cached[64][5] = {};
    int dev = 0;
    check(cudaGetDevice(&dev), "cudaGetDevice");
    ensure_smem<kHistExactConst>();
    ensure_smem<kHistExactVar>();
    ensure_smem<kHistQ16Const>();
    ensure_smem<kHistQ16Var>();
    ensure_smem<kHistQ8Const>();
    ensure_smem<kHistQ8Var>();
    cluster = cluster >= 4 ? 4 : cluster >= 2 ? 2 : 1;
    if (dev >= 0 && dev < 64 && cached[dev][cluster] > 0) return cached[dev][cluster];
    auto kern = wave_hist_kernel<kHistExactConst>;  // the largest shared-memory footprint
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(1, cluster * 64, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = SmemLayout<kHistExactConst>::bytes;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = cluster;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess || clusters <= 0) {
        (void)cudaGetLastError();
        clusters = 148 / cluster;
    }
    if (dev >= 0 && dev < 64) cached[dev][cluster] = clusters;
    return clusters;
}

bool encode_codes_map(CUtensorMap* map, const uint8_t* codes, long long n_rows, int stride) {
    std::memset(map, 0, sizeof(*map));
    if (codes == nullptr || n_rows <= 0 || n_rows > 0x7fffffffll || stride < kFG || stride % 16 != 0 ||
        (reinterpret_cast<uintptr_t>(codes) & 15u) != 0)
        return false;
    using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode encode = [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            (void)cudaGetLastError();
            return static_cast<Encode>(nullptr);
        }
        return reinterpret_cast<Encode>(fn);
    }();
    if (encode == nullptr) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(stride), static_cast<cuuint64_t>(n_rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(stride)};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(kFG), 1u};  // gather4: one row high
    const cuuint32_t elem[2] = {1u, 1u};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(codes), dims, strides, box,
                              elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                              CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        std::memset(map, 0, sizeof(*map));
        return false;
    }
    return true;
}

void launch_wave_hist(int mode, const WaveCtx* ctxs, int n_ctx, int src, HistTune tune,
                      unsigned long long* rows_counter, cudaStream_t s) {
    switch (mode) {
        case kHistExactConst: hist_launch<kHistExactConst>(ctxs, n_ctx, src, tune, rows_counter, s); break;
        case kHistExactVar: hist_launch<kHistExactVar>(ctxs, n_ctx, src, tune, rows_counter, s); break;
        case kHistQ16Const: hist_launch<kHistQ16Const>(ctxs, n_ctx, src, tune, rows_counter, s); break;
        case kHistQ16Var: hist_launch<kHistQ16Var>(ctxs, n_ctx, src, tune, rows_counter, s); break;
        case kHistQ8Const: hist_launch<kHistQ8Const>(ctxs, n_ctx, src, tune, rows_counter, s); break;
        default: hist_launch<kHistQ8Var>(ctxs, n_ctx, src, tune, rows_counter, s); break;
    }
}

void launch_rows_max(const int32_t* rows, int n_rows, const double* g, const double* h, AllScale* sc,
                     cudaStream_t s) {
    if (n_rows <= 0) return;
    rows_max_kernel<<<std::max(1, std::min(1184, (n_rows + 255) / 256)), 256, 0, s>>>(rows, n_rows, g, h, sc);
    check(cudaGetLastError(), "rows_max launch");
}

void launch_wave_partition(const WaveCtx* ctxs, int n_ctx, int grid, bool pair, cudaStream_t s) {
    launch_pdl(pair ? wave_part_kernel<true> : wave_part_kernel<false>, dim3(grid), dim3(kPartThreads), 0, s, "wave_part launch", ctxs, n_ctx);
}

void launch_wave_begin(const WaveBegin& a, cudaStream_t s) {
    wave_begin_kernel<<<148 * 2, 256, 0, s>>>(a);
    check(cudaGetLastError(), "wave_begin launch");
}

void launch_wave_scales(DevTreeState* st, const AllScale* all, int mode, cudaStream_t s) {
    wave_scales_kernel<<<1, 1, 0, s>>>(st, all, mode);
    check(cudaGetLastError(), "wave_scales launch");
}

void launch_wave_quantize(int mode, const int32_t* rows, const double* g, const double* h, const uint8_t* goss_flag,
                          double goss_scale, const DevTreeState* st, unsigned long long seed, bool per_tree, void* gq,
                          void* hq, unsigned long long* energy, int max_rows, cudaStream_t s) {
    const int blocks = std::max(1, std::min(1184, (max_rows + 255) / 256));
    switch (mode) {
        case kHistExactConst: quantize_launch<kHistExactConst>(rows, g, h, goss_flag, goss_scale, st, seed, per_tree, gq, hq, energy, blocks, s); break;
        case kHistExactVar: quantize_launch<kHistExactVar>(rows, g, h, goss_flag, goss_scale, st, seed, per_tree, gq, hq, energy, blocks, s); break;
        case kHistQ16Const: quantize_launch<kHistQ16Const>(rows, g, h, goss_flag, goss_scale, st, seed, per_tree, gq, hq, energy, blocks, s); break;
        case kHistQ16Var: quantize_launch<kHistQ16Var>(rows, g, h, goss_flag, goss_scale, st, seed, per_tree, gq, hq, energy, blocks, s); break;
        case kHistQ8Const: quantize_launch<kHistQ8Const>(rows, g, h, goss_flag, goss_scale, st, seed, per_tree, gq, hq, energy, blocks, s); break;
        default: quantize_launch<kHistQ8Var>(rows, g, h, goss_flag, goss_scale, st, seed, per_tree, gq, hq, energy, blocks, s); break;
    }
    check(cudaGetLastError(), "wave_quantize launch");
}

}  // namespace tgb
