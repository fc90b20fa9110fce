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
// rows: 442 -> 347 us; FP64 alone is about 160).  kGradRoom pairs of room a warp keep seven
// CTAs on an SM; a run of larger classes gives a warp the room of several.
constexpr int kClassRows = 48;
constexpr int kGradRoom = 29 * 28 / 2;
constexpr int kGradWarps = 4;
static_assert(kGradWarps * kGradRoom >= kClassRows * (kClassRows - 1) / 2, "room for the largest class");

__global__ void __launch_bounds__(kGradWarps * 32)
    grad_pairwise_kernel(const double* __restrict__ y, const double* __restrict__ pred,
                         const int* __restrict__ run_start, const int* __restrict__ run_len,
                         const int* __restrict__ order, double* __restrict__ g,
                         double* __restrict__ h, AllScale* __restrict__ sc) {
    double mg = 0.0, mh = 0.0;
    __shared__ double2 s_terms[kGradWarps * kGradRoom];  // {lambda, hessian} of pair b (b - 1) / 2 + a, a < b
    __shared__ double2 s_rows[kGradWarps][kClassRows];   // {y, pred}
    __shared__ unsigned short s_ab[kClassRows * (kClassRows - 1) / 2];  // a | b << 8
    const int r = blockIdx.x;
    const int s0 = run_start[r], m = run_len[r];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int step = m > 48 ? max(1, m / 24) : 1;
    const int most = (m + step - 1) / step;  // rows of class 0, the largest
    for (int b = threadIdx.x; b < most; b += kGradWarps * 32)
        for (int a = 0; a < b; ++a) s_ab[b * (b - 1) / 2 + a] = static_cast<unsigned short>(a | b << 8);
    __syncthreads();
    const int span = max(1, (most * (most - 1) / 2 + kGradRoom - 1) / kGradRoom);  // warps' room a class takes
    const int warps = kGradWarps / span;
    double2 *terms = s_terms + warp * span * kGradRoom, *cls = s_rows[warp];
    for (int c = warp < warps ? warp : m; c < step && c < m; c += warps) {
        const int K = (m - c + step - 1) / step, n_pairs = K * (K - 1) / 2;
        int row[2];
        bool nan = false;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int a = lane + 32 * q;
            row[q] = a < K ? row_at(order, s0 + c + a * step) : -1;
            if (row[q] >= 0) {
                const double ya = y[row[q]];
                cls[a] = make_double2(ya, pred[row[q]]);
                nan |= ya != ya;
            }
        }
        __syncwarp();
        if (__any_sync(0xffffffffu, nan)) {
            // a NaN target is the lower one of its pair for both rows: no shared terms
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int a = lane + 32 * q;
                if (row[q] < 0) continue;
                const double2 A = cls[a];
                double ga = 0.0, ha = 1e-6, l, d;
                for (int b = 0; b < K; ++b) {
                    const double2 B = cls[b];
                    if (b == a || A.x == B.x) continue;
                    const bool a_hi = A.x > B.x;
                    pair_terms(a_hi ? A.y : B.y, a_hi ? B.y : A.y, a_hi ? A.x - B.x : B.x - A.x, l, d);
                    ga += a_hi ? l : -l;
                    ha += d;
                }
                g[row[q]] = ga;
                h[row[q]] = ha;
                mg = fmax(mg, fabs(ga));
                mh = fmax(mh, fabs(ha));
            }
            __syncwarp();
            continue;
        }
        for (int q = lane; q < n_pairs; q += 32) {
            const unsigned ab = s_ab[q];
            const double2 A = cls[ab & 0xffu], B = cls[ab >> 8];
            const bool a_hi = A.x > B.x;
            double l, d;
            pair_terms(a_hi ? A.y : B.y, a_hi ? B.y : A.y, a_hi ? A.x - B.x : B.x - A.x, l, d);
            if (!a_hi) l = -l;  // row a is the lower one
            if (A.x == B.x) l = d = 0.0;
            terms[q] = make_double2(l, d);
        }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int a = lane + 32 * q;
            if (row[q] < 0) continue;
            double ga = 0.0, ha = 1e-6;
            // partners below a: a is the pair's second row; above: its first
            int at = a * (a - 1) / 2;
            for (int b = 0; b < K; ++b) {
                if (b == a) at = a * (a + 1) / 2 + a;  // the pair (a, a + 1)
                else {
                    const double2 t = terms[at];
                    ga += b < a ? -t.x : t.x;
                    ha += t.y;
                    at += b < a ? 1 : b;
                }
            }
            g[row[q]] = ga;
            h[row[q]] = ha;
            mg = fmax(mg, fabs(ga));
            mh = fmax(mh, fabs(ha));
        }
        __syncwarp();
    }
    if (sc != nullptr) block_max_into(mg, mh, sc);
}

__global__ void loss_pairwise_kernel(const double* __restrict__ y, const double* __restrict__ pred,
                                     const int* __restrict__ run_start, const int* __restrict__ run_len,
                                     const int* __restrict__ order, double* __restrict__ corr,
                                     int* __restrict__ valid, int* __restrict__ ticket, DevTreeState* __restrict__ st,
                                     double* __restrict__ losses) {
    const int r = blockIdx.x;
    const int s0 = run_start[r], m = run_len[r];
    __shared__ double red[3][32];
    __shared__ double mean[2];
    __shared__ int s_last;
    double sy = 0, sp = 0;
    for (int k = threadIdx.x; k < m; k += blockDim.x) {
        const int i = row_at(order, s0 + k);
        sy += y[i];
        sp += pred[i];
    }
    for (int o = 16; o > 0; o >>= 1) {
        sy += __shfl_xor_sync(0xffffffffu, sy, o);
        sp += __shfl_xor_sync(0xffffffffu, sp, o);
    }
    const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if ((threadIdx.x & 31) == 0) {
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
    for (int k = threadIdx.x; k < m; k += blockDim.x) {
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
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
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
        s_last = atomicAdd(ticket, 1) == static_cast<int>(gridDim.x) - 1;
        __threadfence();
    }
    __syncthreads();
    if (!s_last) return;
    // the last run to finish: minus the mean correlation over the valid runs, added in a fixed order
    double t = 0.0;
    int n_ok = 0;
    for (int k = threadIdx.x; k < static_cast<int>(gridDim.x); k += blockDim.x)
        if (__ldcg(valid + k)) {
            t += __ldcg(corr + k);
            n_ok += 1;
        }
    for (int o = 16; o > 0; o >>= 1) {
        t += __shfl_xor_sync(0xffffffffu, t, o);
        n_ok += __shfl_xor_sync(0xffffffffu, n_ok, o);
    }
    if ((threadIdx.x & 31) == 0) {
        red[0][w] = t;
        red[1][w] = static_cast<double>(n_ok);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0, k_ok = 0;
        for (int k = 0; k < nw; ++k) {
            a += red[0][k];
            k_ok += red[1][k];
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

void launch_grad_pairwise(const double* y, const double* pred, const int* run_start, const int* run_len,
                          const int* order, int n_runs, int n, double* g, double* h, AllScale* sc, cudaStream_t s) {
    (void)n;
    if (n_runs <= 0) return;
    grad_pairwise_kernel<<<n_runs, kGradWarps * 32, 0, s>>>(y, pred, run_start, run_len, order, g, h, sc);
    check(cudaGetLastError(), "grad_pairwise launch");
}

void launch_loss_pairwise(const double* y, const double* pred, const int* run_start, const int* run_len,
                          const int* order, int n_runs, double* corr, int* valid, int* ticket, DevTreeState* st,
                          double* losses, cudaStream_t s) {
    if (n_runs <= 0) return;
    loss_pairwise_kernel<<<n_runs, 128, 0, s>>>(y, pred, run_start, run_len, order, corr, valid, ticket, st,
                                                losses);
    check(cudaGetLastError(), "loss_pairwise launch");
}

}  // namespace tgb
