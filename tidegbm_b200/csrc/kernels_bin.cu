// Quantile-bin transform: X (row-major f32 or f64) -> uint8 codes, row-major
// [n][stride].  Restates Binner::transform (cpp/src/binning.cpp:104-128):
// code = 1 + upper_bound(edges, v), NaN -> 0 (kMissingBin, cpp/include/tidegbm/types.hpp:20);
// a categorical feature's code is 1 + the value's vocabulary index (0 when absent).
//
// For f32 input the edges arrive as ceil_f32(edge) (the smallest float >= the f64
// edge): for a float v, v < e  <=>  v < ceil_f32(e) (a NaN edge stays NaN), so the float
// compare gives the reference's f64 upper_bound exactly.  f64 input compares against f64
// edges.
//
// Launch shape: one CTA = 8 warps x a group of at most 32 features, and as many CTAs as the
// chip holds at once, each over one contiguous share of the rows (the group's edges are
// staged once per CTA).  A lane owns a feature; a group of fewer features gives a warp
// several rows at a time.  The group's edges sit in shared memory as [edge][lane], so a
// lane only ever reads its own bank: the bisection's probes of a warp are one wavefront each
// whatever the values are.  (With [feature][edge] rows the 32 probes of a step fell on random
// banks, 3.4 deep on average, one row at a time: 2,513 us for 4M x 128 float32.)  Eight rows
// are searched together while the next eight load, and the first two of the eight steps
// compare with edges held in registers, so a value costs six shared loads, compares and
// predicated adds: 805 us there.  Edges past the last are NaN, which no value counts, and rows
// are addressed by uniform pointers and a lane's 32-bit offset: 37 instructions a value instead
// of 41, and registers for a fifth CTA on every SM: 750 us, with issue slots 73% busy and
// waits for X the rest (its bytes take 396 us; four CTAs 805, six of six rows 862).
#include "tgb_internal.h"

#include <cmath>

namespace tgb {

namespace {

constexpr int kBinWarps = 8;
constexpr int kBinThreads = kBinWarps * 32;
constexpr int kBinRows = 8;  // rows a lane searches together
// CTAs per SM: 51 registers a thread, or 64 KB of double edges
constexpr int kBinCtas32 = 5, kBinCtas64 = 3;

// std::upper_bound's own bisection (libstdc++ __upper_bound) over edge k at e[32 k]: the same
// probes and the same answer as the reference, also when NaN edges break the order.
template <typename T>
__device__ __forceinline__ int upper_bound_exact(const T* e, int ne, T v) {
    int first = 0, len = ne;
    while (len > 0) {
        const int half = len >> 1;
        const int mid = first + half;
        if (v < e[32 * mid]) {
            len = half;
        } else {
            first = mid + 1;
            len = len - half - 1;
        }
    }
    return first;
}

// Categorical (binning.cpp:112-117): 1 + the value's index in the sorted vocabulary
// (std::lower_bound's bisection), 0 when it is not in it.
template <typename T>
__device__ __forceinline__ int vocabulary_code(const T* e, int ne, T v) {
    int first = 0, len = ne;
    while (len > 0) {
        const int half = len >> 1;
        const int mid = first + half;
        if (e[32 * mid] < v) {
            first = mid + 1;
            len = len - half - 1;
        } else {
            len = half;
        }
    }
    return (first < ne && e[32 * first] == v) ? first + 1 : 0;
}

// The edge at shared address p + k rows of 32 (the offset is an immediate of the load).
template <int k>
__device__ __forceinline__ float edge_at(unsigned p, float) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1 + %2];" : "=f"(v) : "r"(p), "n"(k * 128));
    return v;
}
template <int k>
__device__ __forceinline__ double edge_at(unsigned p, double) {
    double v;
    asm volatile("ld.shared.f64 %0, [%1 + %2];" : "=d"(v) : "r"(p), "n"(k * 256));
    return v;
}
// p += k if v >= e (never with a NaN), as one compare and one predicated add.
template <unsigned k>
__device__ __forceinline__ void advance(unsigned& p, float v, float e) {
    asm("{ .reg .pred t; setp.ge.f32 t, %1, %2; @t add.u32 %0, %0, %3; }" : "+r"(p) : "f"(v), "f"(e), "n"(k));
}
template <unsigned k>
__device__ __forceinline__ void advance(unsigned& p, double v, double e) {
    asm("{ .reg .pred t; setp.ge.f64 t, %1, %2; @t add.u32 %0, %0, %3; }" : "+r"(p) : "d"(v), "d"(e), "n"(k));
}
// One halving step of kBinRows searches: p is the shared address of the first edge not yet
// known to be <= v.
template <int h, typename T>
__device__ __forceinline__ void halve(unsigned (&p)[kBinRows], const T (&v)[kBinRows]) {
    T e[kBinRows];
#pragma unroll
    for (int q = 0; q < kBinRows; ++q) e[q] = edge_at<h - 1>(p[q], v[q]);
#pragma unroll
    for (int q = 0; q < kBinRows; ++q) advance<h * 32 * sizeof(T)>(p[q], v[q], e[q]);
}

template <typename T>
__global__ void __launch_bounds__(kBinThreads, sizeof(T) == 4 ? kBinCtas32 : kBinCtas64)
    bin_transform_kernel(const T* __restrict__ X, int n, int n_f, const T* __restrict__ edges,
                         const int* __restrict__ n_edges, uint8_t* __restrict__ codes, int stride,
                         int rows_per_cta, const uint8_t* __restrict__ is_cat) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* se = reinterpret_cast<T*>(smem_raw);  // [256][32]
    __shared__ int s_plain[32];
    const int f0 = blockIdx.y * 32;
    const int nf = min(32, n_f - f0);
    const int rpw = 32 / nf;  // rows of a warp's step
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sub = lane / nf, ff = lane - sub * nf;
    const bool active = sub < rpw;
    const int f = f0 + ff;
    const int ne = n_edges[f];
    {
        const T* ef = edges + static_cast<size_t>(f) * 256;
#pragma unroll 1
        for (int b0 = warp; b0 < 256; b0 += 16 * kBinWarps) {
            T v[16];
#pragma unroll
            for (int q = 0; q < 16; ++q) v[q] = b0 + q * kBinWarps < ne ? ef[b0 + q * kBinWarps] : T(NAN);
#pragma unroll
            for (int q = 0; q < 16; ++q) se[(b0 + q * kBinWarps) * 32 + lane] = v[q];
        }
    }
    if (threadIdx.x < 32) s_plain[threadIdx.x] = ne <= 255 ? 1 : 0;
    __syncthreads();
    const T* e = se + lane;
    // ascending edges without NaN: counting the edges <= v by halving steps is upper_bound
    bool plain = true;
#pragma unroll 8
    for (int b = warp; b < 255; b += kBinWarps) {  // past ne the staged edges are NaN: no value counts them
        const T lo = e[32 * b], hi = e[32 * (b + 1)];
        plain &= b >= ne || (b + 1 < ne ? lo <= hi : lo == lo);
    }
    if (!plain) s_plain[lane] = 0;
    __syncthreads();
    plain = s_plain[lane] != 0;
    const bool cat = is_cat != nullptr && is_cat[f] != 0;
    const int r0 = blockIdx.x * rows_per_cta;
    const int r1 = min(n, r0 + rows_per_cta);
    const T e127 = e[32 * 127], e63 = e[32 * 63], e191 = e[32 * 191];
    const int step = kBinWarps * rpw;
    constexpr unsigned kRow = 32 * sizeof(T);  // bytes from one edge to the next
    const unsigned base = static_cast<unsigned>(__cvta_generic_to_shared(e));
    const size_t x_step = static_cast<size_t>(step) * n_f, c_step = static_cast<size_t>(step) * stride;
    int r = r0 + warp * rpw + sub;
    if (active && plain && !cat) {
        // the CTA's rows by uniform pointers, a lane's place in them by a 32-bit offset
        const T* xb = X + static_cast<size_t>(r0) * n_f;
        uint8_t* ob = codes + static_cast<size_t>(r0) * stride;
        const unsigned xo = static_cast<unsigned>(warp * rpw + sub) * n_f + f;
        const unsigned oo = static_cast<unsigned>(warp * rpw + sub) * stride + f;
        const unsigned first = (base / kRow) - 1u;  // code = p / kRow - first
        T nv[kBinRows];  // the next rows' values, loaded while these are searched
        int left = (r1 - r0) / (kBinRows * step);
#pragma unroll
        for (int q = 0; q < kBinRows; ++q) nv[q] = left > 0 ? __ldcs(xb + q * x_step + xo) : T(0);
        r += left * kBinRows * step;
        for (; left > 0; --left, ob += kBinRows * c_step) {
            T v[kBinRows];
            unsigned p[kBinRows];
#pragma unroll
            for (int q = 0; q < kBinRows; ++q) v[q] = nv[q];
            xb += kBinRows * x_step;
            if (left > 1) {
#pragma unroll
                for (int q = 0; q < kBinRows; ++q) nv[q] = __ldcs(xb + q * x_step + xo);
            }
#pragma unroll
            for (int q = 0; q < kBinRows; ++q) {
                p[q] = base;
                advance<128 * kRow>(p[q], v[q], e127);
                advance<64 * kRow>(p[q], v[q], v[q] >= e127 ? e191 : e63);
            }
            halve<32>(p, v);
            halve<16>(p, v);
            halve<8>(p, v);
            halve<4>(p, v);
            halve<2>(p, v);
            halve<1>(p, v);
#pragma unroll
            for (int q = 0; q < kBinRows; ++q)
                (ob + q * c_step)[oo] = static_cast<uint8_t>(v[q] != v[q] ? 0u : p[q] / kRow - first);  // NaN -> 0
        }
    }
    const T* x = X + static_cast<size_t>(r) * n_f + f;
    uint8_t* out = codes + static_cast<size_t>(r) * stride + f;
    if (active) {  // the last rows of a plain feature, all rows of the others
        for (; r < r1; r += step, x += x_step, out += c_step) {
            const T v = *x;
            const int code = cat ? vocabulary_code(e, ne, v) : upper_bound_exact(e, ne, v) + 1;
            *out = static_cast<uint8_t>(v != v ? 0 : code);
        }
    }
    // Zero the padding bytes [n_f, stride) so gathers of whole rows see 0.
    const int pad = stride - n_f;
    if (pad > 0 && blockIdx.y == gridDim.y - 1) {
        const long long total = static_cast<long long>(r1 - r0) * pad;
        for (long long k = threadIdx.x; k < total; k += kBinThreads)
            codes[static_cast<size_t>(r0 + k / pad) * stride + n_f + k % pad] = 0;
    }
}

// Column-major copy for the partition's single-feature reads: a CTA moves a tile of
// 128 rows x 32 features through shared memory (16-byte loads of row chunks, 16-byte
// stores of column runs).
// col has a row pitch of round_up(n, 16) bytes, so every 16-row run is 16-byte aligned.
__global__ void __launch_bounds__(256)
    codes_transpose_kernel(const uint8_t* __restrict__ codes, int stride, int n, int n_f, uint8_t* __restrict__ col,
                           long long pitch) {
    __shared__ uint8_t tile[128][33];
    const int r0 = blockIdx.x * 128, f0 = blockIdx.y * 32;
    {
        const int r = threadIdx.x >> 1, half = threadIdx.x & 1;  // 2 x 16 bytes per row
        const int fb = f0 + half * 16;
        if (r0 + r < n && fb < stride) {
            const uint4 v = *reinterpret_cast<const uint4*>(codes + static_cast<size_t>(r0 + r) * stride + fb);
            const uint8_t* b = reinterpret_cast<const uint8_t*>(&v);
#pragma unroll
            for (int i = 0; i < 16; ++i) tile[r][half * 16 + i] = b[i];
        }
    }
    __syncthreads();
    const int fl = threadIdx.x >> 3, q = threadIdx.x & 7;  // feature, run of 16 rows
    const int f = f0 + fl;
    if (f >= n_f) return;
    const int rb = r0 + q * 16;
    if (rb + 16 <= n) {
        uint4 v;
        uint8_t* b = reinterpret_cast<uint8_t*>(&v);
#pragma unroll
        for (int i = 0; i < 16; ++i) b[i] = tile[q * 16 + i][fl];
        *reinterpret_cast<uint4*>(col + static_cast<size_t>(f) * pitch + rb) = v;
    } else {
        for (int i = 0; i < 16 && rb + i < n; ++i) col[static_cast<size_t>(f) * pitch + rb + i] = tile[q * 16 + i][fl];
    }
}

template <typename T>
void launch_bin(const T* X, int n, int n_f, const T* edges, const int* n_edges, uint8_t* codes,
                int stride, cudaStream_t s, const uint8_t* is_cat) {
    if (n <= 0 || n_f <= 0) return;
    const int groups = (n_f + 31) / 32;
    const size_t smem = sizeof(T) * 32 * 256;
    auto kern = bin_transform_kernel<T>;
    // every CTA resident at once, of at least one step of all warps
    const int ctas = std::max(1, 148 * (sizeof(T) == 4 ? kBinCtas32 : kBinCtas64) / groups);
    const int min_rows = kBinWarps * kBinRows;
    const int rows_per_cta = std::max(min_rows, (n + ctas - 1) / ctas);
    // on every call (under 1 us), so that it holds after a cudaDeviceReset too
    check(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)), "bin smem attr");
    dim3 grid((n + rows_per_cta - 1) / rows_per_cta, groups);
    kern<<<grid, kBinThreads, smem, s>>>(X, n, n_f, edges, n_edges, codes, stride, rows_per_cta, is_cat);
    check(cudaGetLastError(), "bin_transform launch");
}

}  // namespace

void launch_codes_transpose(const uint8_t* codes, int stride, int n, int n_f, uint8_t* col, cudaStream_t s) {
    if (n <= 0 || n_f <= 0) return;
    dim3 grid((n + 127) / 128, (n_f + 31) / 32);
    codes_transpose_kernel<<<grid, 256, 0, s>>>(codes, stride, n, n_f, col, codes_col_pitch(n));
    check(cudaGetLastError(), "codes_transpose launch");
}

void launch_bin_transform_f32(const float* X, int n, int n_f, const float* edges, const int* n_edges,
                              uint8_t* codes, int stride, cudaStream_t s, const uint8_t* is_cat) {
    launch_bin<float>(X, n, n_f, edges, n_edges, codes, stride, s, is_cat);
}

void launch_bin_transform_f64(const double* X, int n, int n_f, const double* edges, const int* n_edges,
                              uint8_t* codes, int stride, cudaStream_t s, const uint8_t* is_cat) {
    launch_bin<double>(X, n, n_f, edges, n_edges, codes, stride, s, is_cat);
}

}  // namespace tgb
