// Gradients/hessians and training losses.
//
// MSE restates Objective::grad_hess (cpp/src/objective.cpp:105-118) with unit
// weights: g = pred - y, h = 1.
//
// RankPairwise restates objective.cpp:179-219.  Per date group of m rows (group_runs,
// objective.cpp:18-39): step = m > 48 ? max(1, m/24) : 1 and pairs (a, a + k*step).
// A row's partners are exactly the positions a -/+ k*step, so a row sums its own pair terms
// (gather, no atomics).  Visiting the partners in ascending position order reproduces the
// reference's accumulation order for that row (contributions as the later element of a pair
// arrive first, for smaller a), so g and h follow the same FP64 addition sequence; this
// file is compiled with -fmad=false to keep the statement-order rounding.
//
// Losses restate Objective::loss (objective.cpp:262-329): mean squared error, and
// for ranking the negative mean within-group Pearson correlation.
#include "tgb_internal.h"

namespace tgb {

namespace {

__global__ void grad_mse_kernel(const double* __restrict__ y, const double* __restrict__ pred, int n,
                                double* __restrict__ g, double* __restrict__ h) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        g[i] = 1.0 * (pred[i] - y[i]);
        h[i] = 1.0;
    }
}

// The MSE gradient fused with the all-row maxima the fit needs from it: g = pred - y
// (the unit hessian is implicit), max |g| and max h = 1 for the all-row fixed-point scale.
__global__ void grad_mse_fused_kernel(const double* __restrict__ y, const double* __restrict__ pred, int n,
                                      double* __restrict__ g, AllScale* __restrict__ sc) {
    double mg = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double gv = 1.0 * (pred[i] - y[i]);
        g[i] = gv;
        mg = fmax(mg, fabs(gv));
    }
    block_max_into(mg, 1.0, sc);
}

__device__ __forceinline__ int row_at(const int* order, int p) { return order ? order[p] : p; }

// One pair of rows of unlike targets (objective.cpp:196-212): the lambda added to the row of
// the larger target and subtracted from the other, and the hessian both get.
__device__ __forceinline__ void pair_terms(double phi, double plo, double dy, double& lam, double& d2) {
    const double s = phi - plo;
    const double e = exp(fmin(fmax(1.0 * s, -30.0), 30.0));
    const double dyw = fmax(fabs(dy), 1e-6);
    lam = -1.0 / (1.0 + e) * dyw;
    d2 = 1.0 * 1.0 * e / ((1 + e) * (1 + e)) * dyw;
}

// A row's partners are the rows of its residue class modulo step, so a class of K rows is a
// clique of K (K - 1) / 2 pairs (K <= 48; at most 36 where m > 48, 24 to 29 from m = 120 on).
// A warp takes a class: lanes evaluate its pairs once each and leave the signed lambda of the
// pair's first row and the hessian in shared memory; then a lane per row adds its row's terms
// in ascending partner order, the order and the terms of the reference, so the sums are the
// same to the last bit (a pair of equal targets leaves zeros, which change no sum).  The
// kernel is bound by instruction issue, most of it the exponential and two FP64 divisions of
// a pair, which are evaluated once instead of once for each row (8,000 dates of 50 to 800
// rows: 442 -> 334 us; FP64 alone is about 160).  kGradRoom pairs of room a warp keep seven
// CTAs on an SM; the warps of a CTA work together on a run of one class, and in twos on larger
// ones and on a run's two (3,000 runs of 48 rows: 65 us with three warps idle, 36 so; of 49: 27, 23).
// A class of equal targets, which has no terms, takes one vote.
constexpr int kClassRows = 48;
constexpr int kGradRoom = 29 * 28 / 2;
constexpr int kGradWarps = 4;
constexpr int kShortRun = 29;  // rows of a run that fit a warp's room
static_assert(kGradWarps * kGradRoom >= kClassRows * (kClassRows - 1) / 2, "room for the largest class");
static_assert(2 * kGradRoom >= 36 * 35 / 2, "two warps' room for the largest of several classes");

// The pairs (a, b), a < b, as a | b << 8 at b (b - 1) / 2 + a: a class of any size uses the first of them.
struct alignas(16) PairTable {
    unsigned short ab[kClassRows * (kClassRows - 1) / 2];
    constexpr PairTable() : ab() {
        for (int b = 1; b < kClassRows; ++b)
            for (int a = 0; a < b; ++a) ab[b * (b - 1) / 2 + a] = static_cast<unsigned short>(a | b << 8);
    }
};
__device__ constexpr PairTable kPairTable;
static_assert(sizeof(PairTable) % 16 == 0, "copied in 16-byte words");

// The first n_pairs entries into shared memory (the caller synchronises the CTA).
__device__ __forceinline__ void copy_pairs(uint4* to, int n_pairs) {
    const uint4* from = reinterpret_cast<const uint4*>(kPairTable.ab);
    for (int k = threadIdx.x; k < (n_pairs + 7) / 8; k += blockDim.x) to[k] = __ldg(from + k);
}

// Gradients of one class, rows s0 + c + a * step for a < K, by `ways` warps of which this one is
// number `part`; terms: their room, cls: this warp's {y, pred} of every row of the class; sync:
// a barrier of those warps.
template <typename Sync>
__device__ __forceinline__ void class_gradients(const double* __restrict__ y, const double* __restrict__ pred,
                                                const int* __restrict__ order, int s0, int c, int step, int K, int part,
                                                int ways, const unsigned short* s_ab, double2* terms, double2* cls, Sync sync,
                                                double* __restrict__ g, double* __restrict__ h, double& mg, double& mh) {
    const int lane = threadIdx.x & 31, mine = lane + 32 * part;
    int row = -1;  // of element `mine`, whose sums this lane makes
    bool nan = false, unlike = false;
    double y0 = 0.0;
    for (int a = lane; a < ((K + 31) & ~31); a += 32) {
        double ya = 0.0;
        if (a < K) {
            const int r = row_at(order, s0 + c + a * step);
            ya = y[r];
            cls[a] = make_double2(ya, pred[r]);
            if (a == mine) row = r;
        }
        if (a == lane) y0 = __shfl_sync(0xffffffffu, ya, 0);
        nan |= ya != ya;
        unlike |= a < K && ya != y0;
    }
    if (!__any_sync(0xffffffffu, unlike)) {  // no pair of unlike targets
        if (row >= 0) {
            g[row] = 0.0;
            h[row] = 1e-6;
            mh = fmax(mh, 1e-6);
        }
        return;
    }
    __syncwarp();
    if (__any_sync(0xffffffffu, nan)) {
        // a NaN target is the lower one of its pair for both rows: no shared terms
        if (row >= 0) {
            const double2 A = cls[mine];
            double ga = 0.0, ha = 1e-6, l, d;
            for (int b = 0; b < K; ++b) {
                const double2 B = cls[b];
                if (b == mine || A.x == B.x) continue;
                const bool a_hi = A.x > B.x;
                pair_terms(a_hi ? A.y : B.y, a_hi ? B.y : A.y, a_hi ? A.x - B.x : B.x - A.x, l, d);
                ga += a_hi ? l : -l;
                ha += d;
            }
            g[row] = ga;
            h[row] = ha;
            mg = fmax(mg, fabs(ga));
            mh = fmax(mh, fabs(ha));
        }
        __syncwarp();
        return;  // every warp of the class has seen the same targets
    }
    const int n_pairs = K * (K - 1) / 2;
    for (int q = mine; q < n_pairs; q += 32 * ways) {
        const unsigned ab = s_ab[q];
        const double2 A = cls[ab & 0xffu], B = cls[ab >> 8];
        const bool a_hi = A.x > B.x;
        double l, d;
        pair_terms(a_hi ? A.y : B.y, a_hi ? B.y : A.y, a_hi ? A.x - B.x : B.x - A.x, l, d);
        if (!a_hi) l = -l;  // row a is the lower one
        if (A.x == B.x) l = d = 0.0;
        terms[q] = make_double2(l, d);
    }
    sync();
    if (row >= 0) {
        double ga = 0.0, ha = 1e-6;
        // partners below: this is the pair's second row; above: its first
        int at = mine * (mine - 1) / 2;
        for (int b = 0; b < K; ++b) {
            if (b == mine) at = mine * (mine + 1) / 2 + mine;  // the pair (mine, mine + 1)
            else {
                const double2 t = terms[at];
                ga += b < mine ? -t.x : t.x;
                ha += t.y;
                at += b < mine ? 1 : b;
            }
        }
        g[row] = ga;
        h[row] = ha;
        mg = fmax(mg, fabs(ga));
        mh = fmax(mh, fabs(ha));
    }
    sync();
}

// kLanes 0: a CTA a run.  Else panels of many short runs, a CTA of which leaves most of its lanes
// without work: 32 / kLanes runs a warp, those of at most kLanes = 8 rows with a lane a row that
// evaluates all of its row's pairs, others of up to kShortRun rows by the warp, longer ones by
// the CTA, one by one.
template <int kLanes>
__global__ void __launch_bounds__(kGradWarps * 32)
    grad_pairwise_kernel(const double* __restrict__ y, const double* __restrict__ pred,
                         const int* __restrict__ run_start, const int* __restrict__ run_len,
                         const int* __restrict__ order, int n_runs, double* __restrict__ g,
                         double* __restrict__ h, AllScale* __restrict__ sc) {
    double mg = 0.0, mh = 0.0;
    __shared__ double2 s_terms[kGradWarps * kGradRoom];  // {lambda, hessian} of a pair
    __shared__ double2 s_rows[kGradWarps][kClassRows];   // {y, pred}
    __shared__ uint4 s_pairs[sizeof(PairTable) / 16];
    const unsigned short* s_ab = reinterpret_cast<const unsigned short*>(s_pairs);
    const int warp = threadIdx.x >> 5;
    auto whole_run = [&](int r) {
        const int s0 = run_start[r], m = run_len[r];
        const int step = m > 48 ? max(1, m / 24) : 1;
        const int most = (m + step - 1) / step;  // rows of class 0, the largest
        copy_pairs(s_pairs, most * (most - 1) / 2);
        __syncthreads();
        const int ways = step == 1 ? 4 : step == 2 || most * (most - 1) / 2 > kGradRoom ? 2 : 1;
        const int group = warp / ways, part = warp - group * ways;
        double2 *terms = s_terms + group * ways * kGradRoom, *cls = s_rows[warp];
        for (int c = group; c < step && c < m; c += kGradWarps / ways) {
            const int K = (m - c + step - 1) / step;
            if (ways == 1)
                class_gradients(y, pred, order, s0, c, step, K, 0, 1, s_ab, terms, cls, [] { __syncwarp(); }, g, h, mg, mh);
            else if (ways == 2)
                class_gradients(y, pred, order, s0, c, step, K, part, 2, s_ab, terms, cls,
                                [&] {
                                    __syncwarp();
                                    if (group == 0) asm volatile("bar.sync 1, 64;" ::: "memory");
                                    else asm volatile("bar.sync 2, 64;" ::: "memory");
                                },
                                g, h, mg, mh);
            else
                class_gradients(y, pred, order, s0, c, step, K, part, 4, s_ab, terms, cls, [] { __syncthreads(); }, g, h, mg,
                                mh);
        }
    };
    if constexpr (kLanes != 0) {
        constexpr int kPer = 32 / kLanes;
        const int r0 = blockIdx.x * kGradWarps * kPer, rw = r0 + warp * kPer;
        copy_pairs(s_pairs, kGradRoom);
        __syncthreads();
        if constexpr (kLanes < 32) {
            const int lane = threadIdx.x & 31, a = lane % kLanes, r = rw + lane / kLanes;
            const int m = r < n_runs ? run_len[r] : 0;
            if (a < m && m <= kLanes) {
                const int s0 = run_start[r], i = row_at(order, s0 + a);
                const double yi = y[i], pi = pred[i];
                double ga = 0.0, ha = 1e-6, l, d;
                for (int b = 0; b < m; ++b) {
                    const int j = row_at(order, s0 + b);
                    const double yj = y[j], pj = pred[j];
                    if (b == a || yi == yj) continue;
                    const bool hi = yi > yj;
                    pair_terms(hi ? pi : pj, hi ? pj : pi, hi ? yi - yj : yj - yi, l, d);
                    ga += hi ? l : -l;
                    ha += d;
                }
                g[i] = ga;
                h[i] = ha;
                mg = fmax(mg, fabs(ga));
                mh = fmax(mh, fabs(ha));
            }
            __syncwarp();
        }
        for (int k = 0; k < kPer && rw + k < n_runs; ++k) {
            const int m = run_len[rw + k];
            if (m > (kLanes < 32 ? kLanes : 0) && m <= kShortRun)
                class_gradients(y, pred, order, run_start[rw + k], 0, 1, m, 0, 1, s_ab, s_terms + warp * kGradRoom,
                                s_rows[warp], [] { __syncwarp(); }, g, h, mg, mh);
        }
        for (int k = 0; k < kGradWarps * kPer && r0 + k < n_runs; ++k) {
            if (run_len[r0 + k] <= kShortRun) continue;
            __syncthreads();
            whole_run(r0 + k);
        }
    } else {
        whole_run(blockIdx.x);
    }
    if (sc != nullptr) block_max_into(mg, mh, sc);
}

// A CTA a run; the last one to finish adds the correlations up, all loads of a step before the
// first use: 100,000 runs of 3 rows 311 us (611 with a load of the correlation behind each load
// of its flag, 128 threads over all of them; 353 with resident CTAs that walk the runs).
constexpr int kLossThreads = 128;
constexpr int kLossSums = 8;  // partial sums a thread of the last CTA: 1,024 in all

__global__ void __launch_bounds__(kLossThreads)
    loss_pairwise_kernel(const double* __restrict__ y, const double* __restrict__ pred,
                         const int* __restrict__ run_start, const int* __restrict__ run_len,
                         const int* __restrict__ order, double* __restrict__ corr,
                         int* __restrict__ valid, int* __restrict__ ticket, DevTreeState* __restrict__ st,
                         double* __restrict__ losses) {
    const int n_runs = gridDim.x, r = blockIdx.x;
    const int s0 = run_start[r], m = run_len[r];
    __shared__ double red[3][32];
    __shared__ double mean[2];
    __shared__ int s_last, s_ok[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = kLossThreads / 32;
    double sy = 0, sp = 0;
    for (int k = threadIdx.x; k < m; k += kLossThreads) {
        const int i = row_at(order, s0 + k);
        sy += y[i];
        sp += pred[i];
    }
    for (int o = 16; o > 0; o >>= 1) {
        sy += __shfl_xor_sync(0xffffffffu, sy, o);
        sp += __shfl_xor_sync(0xffffffffu, sp, o);
    }
    if (lane == 0) {
        red[0][w] = sy;
        red[1][w] = sp;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0, b = 0;
        for (int k = 0; k < nw; ++k) {
            a += red[0][k];
            b += red[1][k];
        }
        mean[0] = a / m;
        mean[1] = b / m;
    }
    __syncthreads();
    double vy = 0, vp = 0, c = 0;
    for (int k = threadIdx.x; k < m; k += kLossThreads) {
        const int i = row_at(order, s0 + k);
        const double dy = y[i] - mean[0], dp = pred[i] - mean[1];
        vy += dy * dy;
        vp += dp * dp;
        c += dy * dp;
    }
    for (int o = 16; o > 0; o >>= 1) {
        vy += __shfl_xor_sync(0xffffffffu, vy, o);
        vp += __shfl_xor_sync(0xffffffffu, vp, o);
        c += __shfl_xor_sync(0xffffffffu, c, o);
    }
    if (lane == 0) {  // (the sums of y and pred were read before the last barrier)
        red[0][w] = vy;
        red[1][w] = vp;
        red[2][w] = c;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0, b = 0, cc = 0;
        for (int k = 0; k < nw; ++k) {
            a += red[0][k];
            b += red[1][k];
            cc += red[2][k];
        }
        const bool ok = m >= 3 && a > 1e-18 && b > 1e-18;
        corr[r] = ok ? cc / sqrt(a * b) : 0.0;
        valid[r] = ok ? 1 : 0;
        __threadfence();
        s_last = atomicAdd(ticket, 1) == n_runs - 1;
        __threadfence();
    }
    __syncthreads();
    if (!s_last) return;
    // The last CTA: minus the mean correlation over the valid runs, added in a fixed order, as 1,024
    // threads over the runs and then their 32 warps would.
    double t[kLossSums] = {};
    int n_ok[kLossSums] = {};
#pragma unroll 2
    for (int k0 = threadIdx.x; k0 < n_runs; k0 += kLossThreads * kLossSums) {
        double c[kLossSums];
        int ok[kLossSums];
#pragma unroll
        for (int q = 0; q < kLossSums; ++q) {  // a run that is not valid has left a zero
            const int k = k0 + q * kLossThreads;
            c[q] = k < n_runs ? __ldcg(corr + k) : 0.0;
            ok[q] = k < n_runs ? __ldcg(valid + k) : 0;
        }
#pragma unroll
        for (int q = 0; q < kLossSums; ++q) {
            t[q] += c[q];
            n_ok[q] += ok[q];
        }
    }
#pragma unroll
    for (int q = 0; q < kLossSums; ++q) {
        for (int o = 16; o > 0; o >>= 1) {
            t[q] += __shfl_xor_sync(0xffffffffu, t[q], o);
            n_ok[q] += __shfl_xor_sync(0xffffffffu, n_ok[q], o);
        }
        if (lane == 0) {
            red[0][q * nw + w] = t[q];
            s_ok[q * nw + w] = n_ok[q];
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0;
        int k_ok = 0;
        for (int k = 0; k < kLossSums * nw; ++k) {
            a += red[0][k];
            k_ok += s_ok[k];
        }
        losses[st->tree] = k_ok > 0 ? -a / k_ok : 0.0;
        *ticket = 0;
        st->tree += 1;  // only this thread reads it here
    }
}

}  // namespace

void launch_grad_mse(const double* y, const double* pred, int n, double* g, double* h, cudaStream_t s) {
    if (n <= 0) return;
    grad_mse_kernel<<<std::min(2368, (n + 255) / 256), 256, 0, s>>>(y, pred, n, g, h);
    check(cudaGetLastError(), "grad_mse launch");
}

void launch_grad_mse_fused(const double* y, const double* pred, int n, double* g, AllScale* sc, cudaStream_t s) {
    check(cudaMemsetAsync(sc, 0, 2 * sizeof(unsigned long long), s), "all scale reset");
    if (n <= 0) return;
    grad_mse_fused_kernel<<<std::min(2368, (n + 255) / 256), 256, 0, s>>>(y, pred, n, g, sc);
    check(cudaGetLastError(), "grad_mse_fused launch");
}

// A CTA a run is best while all of them are resident at once (seven on an SM); from there on short
// runs take a warp each, and where the warps run in many rounds, very short ones share it.  us by a
// CTA / a warp / eight lanes: 592 x 24 rows 8.6 / 8.9 / -, 1,200 x 24 12.8 / 10.4 / 25, 1,200 x 8
// 8.7 / 5.9 / 8.8, 5,000 x 8 17.0 / 8.9 / 8.9, 50,000 x 29 265 / 138 / 152, x 30 271 / 273 / 320,
// x 9 136 / 54 / 48, x 3 116 / 35 / 21 (1,200 x 3 5.9 by a warp, 6.9 by eight lanes).
constexpr int kShortRuns = 148 * 7;
constexpr int kManyRuns = 8192;

void launch_grad_pairwise(const double* y, const double* pred, const int* run_start, const int* run_len,
                          const int* order, int n_runs, int n, double* g, double* h, AllScale* sc, cudaStream_t s) {
    if (n_runs <= 0) return;
    const int rows = n / n_runs;  // of a run, on average
    auto launch = [&](auto kern, int runs_a_cta) {
        kern<<<(n_runs + runs_a_cta - 1) / runs_a_cta, kGradWarps * 32, 0, s>>>(y, pred, run_start, run_len, order, n_runs, g,
                                                                               h, sc);
    };
    if (n_runs <= kShortRuns || rows > kShortRun) launch(grad_pairwise_kernel<0>, 1);
    else if (n_runs < kManyRuns || rows > 8) launch(grad_pairwise_kernel<32>, kGradWarps);
    else launch(grad_pairwise_kernel<8>, kGradWarps * 4);
    check(cudaGetLastError(), "grad_pairwise launch");
}

void launch_loss_pairwise(const double* y, const double* pred, const int* run_start, const int* run_len,
                          const int* order, int n_runs, double* corr, int* valid, int* ticket, DevTreeState* st,
                          double* losses, cudaStream_t s) {
    if (n_runs <= 0) return;
    loss_pairwise_kernel<<<n_runs, kLossThreads, 0, s>>>(y, pred, run_start, run_len, order, corr, valid, ticket, st, losses);
    check(cudaGetLastError(), "loss_pairwise launch");
}

}  // namespace tgb
