// GOSS row selection (cpp/src/booster.cpp:554-585): keep the ceil(top * n) rows of
// largest |g|, plus n_other rows drawn from the rest, whose g and h are scaled by
// (1 - top) / other; the sample is then re-sorted by row index.
//
// The reference orders rows by |g| descending (std::sort), shuffles the remainder with
// the booster's mt19937 (std::shuffle) and keeps the first n_other.  The shuffle's
// swap positions depend only on the generator state and the remainder's length, not
// on the data, so the host derives, per tree, the list rest_pos[p] = "position in the
// |g|-descending remainder of the p-th kept row" (see booster.cpp's sample_positions
// in this library) and the device does the data-dependent part:
//   keys = bit pattern of |g| (non-negative doubles order like their bits), radix
//   sort descending (stable; rows with equal |g| keep index order; the row indices are
//   written once per fit).  The sort runs on a 32-bit order-keeping compression of the
//   pattern (4 radix passes instead of 8) and a fix-up pass re-orders the short runs of
//   tied 32-bit keys by the full pattern, which gives exactly the order of the full
//   64-bit stable sort,
//   flag[order[p]] = 1 for p < n_top, flag[order[n_top + rest_pos[p]]] = 2, with the
//   maxima of the sample's |g| and |h| (as the tree sees them) reduced on the way,
//   compaction of flagged rows in index order -> the tree's root row list.
// The hist kernel multiplies g and h of flag-2 rows by the GOSS scale on the fly.
#include "tgb_internal.h"

#include <cub/device/device_radix_sort.cuh>

namespace tgb {

namespace {

// Sort keys from g: the full |g| bit pattern (exact path), or a 32-bit key that keeps the
// order of the patterns (ties allowed): patterns at or above lo = (e_max - 63) << 52,
// e_max the exponent of max |g| (sc), map to (pattern - lo) >> 26, i.e. 6 exponent and 26
// mantissa bits over the 64 binades below the maximum; smaller values (zeros included)
// map to 0.
template <bool kExact>
__global__ void goss_keys_kernel(const double* __restrict__ g, int n, const AllScale* __restrict__ sc,
                                 void* __restrict__ keys, uint8_t* __restrict__ flag) {
    const unsigned long long e_max = sc->maxg_bits >> 52;
    const unsigned long long lo = e_max >= 63 ? (e_max - 63) << 52 : 0ull;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(fabs(g[i])));
        if (kExact) static_cast<unsigned long long*>(keys)[i] = b;
        else static_cast<unsigned int*>(keys)[i] = b >= lo ? static_cast<unsigned int>((b - lo) >> 26) : 0u;
        flag[i] = 0;  // the mark kernel sets the sample's
    }
}

// After the stable sort by 32-bit keys, rows whose keys tie form runs in index order.
// Every element of a run computes its rank inside the run by the full |g| pattern
// (descending, index ascending on exact ties) and writes itself there in `fixed`, which
// gives the order of the full 64-bit stable sort at the run's positions; positions
// outside runs keep order[] (the mark kernel reads fixed[] only at run positions).  A
// run longer than kMaxRun is already in order when all its patterns are equal (checked
// pairwise); otherwise it sets *overflow (the fit then repeats with the 64-bit sort).
constexpr int kMaxRun = 64;

__device__ __forceinline__ unsigned long long abs_bits(const double* g, int32_t r) {
    return static_cast<unsigned long long>(__double_as_longlong(fabs(g[r])));
}

__device__ __forceinline__ bool in_run(const unsigned int* __restrict__ k32, int p, int n) {
    const unsigned int k = k32[p];
    return (p > 0 && k32[p - 1] == k) || (p + 1 < n && k32[p + 1] == k);
}

__global__ void goss_fixup_kernel(const unsigned int* __restrict__ k32, const int32_t* __restrict__ order,
                                  int32_t* __restrict__ fixed, const double* __restrict__ g, int n,
                                  int* __restrict__ overflow) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        if (!in_run(k32, p, n)) continue;
        const unsigned int k = k32[p];
        const int32_t me = order[p];
        int a = p;
        while (a > 0 && p - a < kMaxRun && k32[a - 1] == k) --a;
        int e = p + 1;
        while (e < n && e - a < kMaxRun && k32[e] == k) ++e;
        const unsigned long long km = abs_bits(g, me);
        if (e - a > kMaxRun || (a > 0 && k32[a - 1] == k) || (e < n && k32[e] == k)) {
            // long run (of kMaxRun + 1 the last element sees the whole): in order as it is only if
            // every pattern in it is equal
            if (p > 0 && k32[p - 1] == k && abs_bits(g, order[p - 1]) != km) atomicExch(overflow, 1);
            fixed[p] = me;
            continue;
        }
        int rank = 0;
        for (int q = a; q < e; ++q) {
            if (q == p) continue;
            const unsigned long long kq = abs_bits(g, order[q]);
            if (kq > km || (kq == km && q < p)) ++rank;  // inside a run, position order is index order
        }
        fixed[a + rank] = me;
    }
}

__global__ void goss_iota_kernel(int32_t* __restrict__ vals, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) vals[i] = i;
}

// The flagged rows (flag 1 or 2) in ascending order, and their number: counts per tile of kFlagTile
// rows, then each tile's rows behind the counts of those before it.  A thread has 16 rows, one
// load; the scatter loads its first tile while the counts are still made.  10M rows, 30% flagged:
// 54 -> 19 us (through the row partition's kernels, a byte a load, before); 1.2M: 12 -> 6.
constexpr int kFlagThreads = 256;
constexpr int kFlagTile = kFlagThreads * 16;

// One bit per flagged row of the 16 from r.
__device__ __forceinline__ unsigned flagged(const uint8_t* __restrict__ flag, int n, long long r) {
    unsigned bits = 0;
    if (r + 16 <= n) {
        const uint4 v = *reinterpret_cast<const uint4*>(flag + r);
        const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) bits |= (((w[q] | w[q] >> 1) & 0x01010101u) * 0x10204080u >> 28) << (4 * q);
    } else {
        for (int q = 0; q < 16 && r + q < n; ++q) bits |= (flag[r + q] != 0 ? 1u : 0u) << q;
    }
    return bits;
}

__device__ __forceinline__ int flag_block_sum(int v, int* red) {
    v = __reduce_add_sync(0xffffffffu, v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    int t = 0;
#pragma unroll
    for (int w = 0; w < kFlagThreads / 32; ++w) t += red[w];
    return t;
}

__global__ void __launch_bounds__(kFlagThreads)
    flag_count_kernel(const uint8_t* __restrict__ flag, int n, int n_tiles, int* __restrict__ tile_counts) {
    pdl_trigger();
    __shared__ int red[kFlagThreads / 32];
    for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
        const int c = flag_block_sum(__popc(flagged(flag, n, static_cast<long long>(t) * kFlagTile + threadIdx.x * 16)), red);
        if (threadIdx.x == 0) tile_counts[t] = c;
    }
}

__global__ void __launch_bounds__(kFlagThreads)
    flag_scatter_kernel(const uint8_t* __restrict__ flag, int n, int n_tiles, const int* __restrict__ tile_counts,
                        int32_t* __restrict__ out, int* __restrict__ n_out) {
    __shared__ int red[kFlagThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned bits = flagged(flag, n, static_cast<long long>(blockIdx.x) * kFlagTile + threadIdx.x * 16);
    pdl_wait();
    if (blockIdx.x == 0) {
        int all = 0;
        for (int k = threadIdx.x; k < n_tiles; k += kFlagThreads) all += tile_counts[k];
        all = flag_block_sum(all, red);
        if (threadIdx.x == 0) *n_out = all;
    }
    int counted = 0, before = 0;  // the rows of the tiles below `counted`
    for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
        int part = 0;
        for (int k = counted + threadIdx.x; k < t; k += kFlagThreads) part += tile_counts[k];
        before += flag_block_sum(part, red);
        counted = t;
        const long long r = static_cast<long long>(t) * kFlagTile + threadIdx.x * 16;
        if (t != static_cast<int>(blockIdx.x)) bits = flagged(flag, n, r);
        const int c = __popc(bits);
        int incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        __syncthreads();
        if (lane == 31) red[warp] = incl;
        __syncthreads();
        int at = before + incl - c;
        for (int w = 0; w < warp; ++w) at += red[w];
        for (unsigned m = bits; m != 0; m &= m - 1) out[at++] = static_cast<int32_t>(r) + __ffs(m) - 1;
    }
}

// Marks the sample and reduces the maxima the histogram scales need over it: |g| and
// |h| of the top rows, |g * scale| and |h * scale| of the sampled others (the values the
// tree sees).  With unit hessians (h == nullptr) the maxima are known from two rows: the
// first of the |g| order (the largest |g|) and the sampled other of smallest remainder
// rank (min_rest, the largest |g| among them); only those two threads read g.
__global__ void goss_mark_kernel(const int32_t* __restrict__ order, const unsigned int* __restrict__ k32,
                                 const int32_t* __restrict__ fixed, int n, int n_top, int n_other,
                                 const int32_t* __restrict__ rest, int rest_words, const double* __restrict__ g,
                                 const double* __restrict__ h, double goss_scale, uint8_t* __restrict__ flag,
                                 DevTreeState* __restrict__ st) {
    const int total = n_top + n_other;
    const int32_t* __restrict__ rest_pos = rest + static_cast<size_t>(st->tree & 1) * rest_words;
    const int min_rest = rest_pos[rest_words - 1];
    double mg = 0.0, mh = 0.0;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < total; p += gridDim.x * blockDim.x) {
        const bool top = p < n_top;
        const int rp = top ? 0 : rest_pos[p - n_top];
        const int pos = top ? p : n_top + rp;
        const int r = (k32 != nullptr && in_run(k32, pos, n)) ? fixed[pos] : order[pos];
        flag[r] = top ? 1 : 2;
        if (h != nullptr) {
            mg = fmax(mg, top ? fabs(g[r]) : fabs(g[r] * goss_scale));
            mh = fmax(mh, top ? fabs(h[r]) : fabs(h[r] * goss_scale));
        } else if (top ? p == 0 : rp == min_rest) {
            mg = fmax(mg, top ? fabs(g[r]) : fabs(g[r] * goss_scale));
            mh = fmax(mh, top ? 1.0 : fabs(1.0 * goss_scale));
        }
    }
    // one atomic a CTA and maximum, where there is one
    __shared__ double s_mg[8], s_mh[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mg = fmax(mg, __shfl_xor_sync(0xffffffffu, mg, o));
        mh = fmax(mh, __shfl_xor_sync(0xffffffffu, mh, o));
    }
    if ((threadIdx.x & 31) == 0) {
        s_mg[threadIdx.x >> 5] = mg;
        s_mh[threadIdx.x >> 5] = mh;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < static_cast<int>(blockDim.x >> 5); ++w) {
            mg = fmax(mg, s_mg[w]);
            mh = fmax(mh, s_mh[w]);
        }
        if (mg > 0.0 || mh > 0.0) {
            atomicMax(&st->max_abs_g_bits, static_cast<unsigned long long>(__double_as_longlong(mg)));
            atomicMax(&st->max_h_bits, static_cast<unsigned long long>(__double_as_longlong(mh)));
        }
    }
}

}  // namespace

size_t goss_cub_bytes(int n, bool exact) {
    size_t bytes = 0;
    if (exact)
        check(cub::DeviceRadixSort::SortPairsDescending(nullptr, bytes, static_cast<unsigned long long*>(nullptr),
                                                        static_cast<unsigned long long*>(nullptr),
                                                        static_cast<int32_t*>(nullptr), static_cast<int32_t*>(nullptr),
                                                        n),
              "cub sizing");
    else
        check(cub::DeviceRadixSort::SortPairsDescending(nullptr, bytes, static_cast<unsigned int*>(nullptr),
                                                        static_cast<unsigned int*>(nullptr),
                                                        static_cast<int32_t*>(nullptr), static_cast<int32_t*>(nullptr),
                                                        n),
              "cub sizing");
    return bytes;
}

void launch_goss_iota(int32_t* vals, int n, cudaStream_t s) {
    goss_iota_kernel<<<std::max(1, std::min(2368, (n + 255) / 256)), 256, 0, s>>>(vals, n);
    check(cudaGetLastError(), "goss_iota launch");
}

void launch_goss_select(const double* g, const double* h, int n, int n_top, int n_other, const int32_t* rest,
                        GossWork& w, const AllScale* all, double goss_scale, uint8_t* goss_flag, int32_t* rows0,
                        int* tile_counts, DevTreeState* st, cudaStream_t s) {
    const int blocks = std::max(1, std::min(2368, (n + 255) / 256));
    if (w.exact) goss_keys_kernel<true><<<blocks, 256, 0, s>>>(g, n, all, w.keys_in, goss_flag);
    else goss_keys_kernel<false><<<blocks, 256, 0, s>>>(g, n, all, w.keys_in, goss_flag);
    check(cudaGetLastError(), "goss_keys launch");
    size_t tmp = w.cub_tmp_bytes;
    if (w.exact) {
        check(cub::DeviceRadixSort::SortPairsDescending(w.cub_tmp, tmp, static_cast<unsigned long long*>(w.keys_in),
                                                        static_cast<unsigned long long*>(w.keys_out), w.vals_in,
                                                        w.vals_out, n, 0, 64, s),
              "goss sort");
    } else {
        check(cub::DeviceRadixSort::SortPairsDescending(w.cub_tmp, tmp, static_cast<unsigned int*>(w.keys_in),
                                                        static_cast<unsigned int*>(w.keys_out), w.vals_in,
                                                        w.vals_out, n, 0, 32, s),
              "goss sort");
        // run positions re-ordered into keys_in's memory (free once sorted)
        goss_fixup_kernel<<<blocks, 256, 0, s>>>(static_cast<const unsigned int*>(w.keys_out), w.vals_out,
                                                  static_cast<int32_t*>(w.keys_in), g, n, w.overflow);
        check(cudaGetLastError(), "goss_fixup launch");
    }
    const unsigned int* k32 = w.exact ? nullptr : static_cast<const unsigned int*>(w.keys_out);
    const int32_t* fixed = static_cast<const int32_t*>(w.keys_in);
    goss_mark_kernel<<<std::max(1, std::min(2368, (n_top + n_other + 255) / 256)), 256, 0, s>>>(
        w.vals_out, k32, fixed, n, n_top, n_other, rest, goss_rest_words(n_other), g, h, goss_scale, goss_flag,
        st);
    check(cudaGetLastError(), "goss_mark launch");
    const int n_tiles = (n + kFlagTile - 1) / kFlagTile;
    const int grid = std::min(n_tiles, 148 * 8);
    flag_count_kernel<<<grid, kFlagThreads, 0, s>>>(goss_flag, n, n_tiles, tile_counts);
    check(cudaGetLastError(), "flag_count launch");
    launch_pdl(flag_scatter_kernel, dim3(grid), dim3(kFlagThreads), 0, s, "flag_scatter launch", goss_flag, n, n_tiles,
               tile_counts, rows0, &st->n_sample);
}

}  // namespace tgb
