// Prefixes of libstdc++'s std::shuffle on the device.
//
// std::shuffle over m >= 2^16 elements with std::mt19937 makes one draw j_t in [0, t]
// per t = 1 .. m-1 and swaps a[t] with a[j_t].  Position t is untouched before step t,
// so the step is a[t] = a[j_t]; a[j_t] = t.  For a kept slot p < keep this gives:
//   - if some step t writes p (j_t = p), the slot ends with the last such t;
//   - otherwise (p > 0) it keeps what step p moved in: the value of slot j_p after
//     step p-1.  "The value of slot q after step s" is again the last t <= s with
//     j_t = q, or, if there is none, the value of slot j_q after step q-1 (slot 0
//     starts as 0).  q falls at every step, and only draws t < keep take part.
// So the prefix needs no sequential swaps:
//   shuffle_draw_kernel     one CTA per range runs the generator: last[j] = max t over
//                           draws j < keep; the head draws (t < keep) also record
//                           head[t] = j and count cnt[j]
//   shuffle_scan_kernel     cnt -> bucket ends (one CTA per range)
//   shuffle_bucket_kernel   bucket q lists the head steps t with j_t = q
//   shuffle_resolve_kernel  every slot: last[p], else the walk above, answered from the
//                           buckets; written over last[p]
// The generator is MT19937 (Matsumoto & Nishimura, ACM TOMACS 8(1), 1998), seeded as
// std::mt19937(seed) is, with the 624-word state in shared memory, two words a thread.
// A refill is the recurrence x[k+624] = x[k+397] ^ mix(x[k], x[k+1]); with
// a[k] = mix(old[k], old[k+1]) (^ old[k+397] for k < 227) the new words are
// a[k] ^ a[k-227] ^ a[k-454] (terms with negative index omitted), and word 623 mixes
// with the new word 0: one shared-memory pass and two barriers per 624 words.
// Word q of a block serves draw t + q.  Lemire's method (the one libstdc++'s
// uniform_int_distribution uses for a 32-bit generator) rejects a word when the low
// half of w * (t + 1) is below 2^32 mod (t + 1); that draw then takes the next word,
// shifting the later ones by one.  Rejections happen with probability below
// (t + 1) / 2^32: one block in three has one at ten million values.  A round tests the words
// that are left for their draws as they stand; the draws before the first rejected word are
// committed, and the words behind it go round again.
// The draws are a chain of blocks on one SM, bound by the latency of its steps.  So ten warps
// run the generator, four blocks ahead of the ten that test and commit; a round covers those
// four blocks and has one barrier; indexes are 32 bits wide; only a warp with a word that may
// be rejected (low half below t + 1) divides; hits on kept slots are predicated reductions; and
// the state and the recurrence's terms are padded with zeros where a word lacks one.  10M draws
// into 200,000 slots: 12.2 -> 7.7 ms (20 warps doing both, four barriers a rejection before).
// A round takes about 1,400 cycles whatever its words, hence four blocks: two take 12.8 ms,
// three 7.4, six 9.3, eight 9.2.
#include "tgb_internal.h"

#include <cub/block/block_scan.cuh>

namespace tgb {

namespace {

constexpr int kMtN = 624;
constexpr int kMtHalf = kMtN / 2;
constexpr int kDrawRole = 320;     // threads of a role, two words of a block each
constexpr int kDrawThreads = 2 * kDrawRole;
constexpr int kDrawBlocks = 4;     // blocks a round
constexpr int kDrawWords = kDrawBlocks * kMtN;
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;

__device__ __forceinline__ uint32_t mt_mix(uint32_t hi, uint32_t lo) {
    const uint32_t y = (hi & 0x80000000u) | (lo & 0x7fffffffu);
    return (y >> 1) ^ ((0u - (y & 1u)) & 0x9908b0dfu);
}

__device__ __forceinline__ uint32_t mt_temper(uint32_t v) {
    v ^= v >> 11;
    v ^= (v << 7) & 0x9d2c5680u;
    v ^= (v << 15) & 0xefc60000u;
    v ^= v >> 18;
    return v;
}

// The threads of one role (the barrier wants whole warps).
__device__ __forceinline__ void role_sync(int id) {
    __syncwarp();
    asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(kDrawRole) : "memory");
}

// Range r: std::mt19937(seeds[r]) and draws t = 1 .. ms[r]-1 (ms[r] = 0: the range is
// not handled here; ms[r] < 2^31).  last/head hold keep entries per range, cnt keep + 1.  A range
// whose refills exceed twice the expected count sets *err and stops.
__global__ void __launch_bounds__(kDrawThreads)
    shuffle_draw_kernel(const uint32_t* __restrict__ seeds, const long long* __restrict__ ms, int keep,
                        int32_t* __restrict__ last, int32_t* __restrict__ head, int32_t* __restrict__ cnt,
                        int* __restrict__ err) {
    __shared__ uint32_t st[kMtN + 96];   // zeros after the state: word k >= 227 has no old[k + 397]
    __shared__ uint32_t az[227 + kMtN];  // zeros before a[]: word k < 227 has no a[k - 227], ...
    __shared__ uint32_t words[2][kDrawWords];
    // The first rejected word, by turns: round k posts in slot k % 3, reads it after the barrier,
    // and clears slot (k + 2) % 3, which every thread had read before that barrier and uses
    // after the next.
    __shared__ int first[3];
    __shared__ int stop[2];  // of even and odd rounds: set in a round for the next, read after its barrier
    const int r = blockIdx.x;
    const long long m64 = ms[r];
    if (m64 < 2 || keep <= 0) return;
    const uint32_t m = static_cast<uint32_t>(m64);
    const bool draws = threadIdx.x < kDrawRole;
    const int t = draws ? threadIdx.x : threadIdx.x - kDrawRole;
    const bool has = t < kMtHalf;  // the words t and t + 312 of a block
    const int t0 = has ? t : 0;    // (the last eight threads of a role only wait)
    for (int k = threadIdx.x; k < 227; k += kDrawThreads) az[k] = 0u;
    for (int k = kMtN + threadIdx.x; k < kMtN + 96; k += kDrawThreads) st[k] = 0u;
    if (threadIdx.x == 0) {  // std::mt19937's seeding recurrence
        uint32_t x = seeds[r];
        st[0] = x;
        for (int k = 1; k < kMtN; ++k) {
            x = 1812433253u * (x ^ (x >> 30)) + static_cast<uint32_t>(k);
            st[k] = x;
        }
        stop[0] = stop[1] = 0;
    }
    if (threadIdx.x < 3) first[threadIdx.x] = kDrawWords;
    __syncthreads();
    uint32_t* a = az + 227;
    auto refill = [&](uint32_t* out) {
        for (int b = 0; b < kDrawBlocks; ++b, out += kMtN) {
            uint32_t a0 = mt_mix(st[t0], st[t0 + 1]) ^ st[t0 + 397];
            const uint32_t hi = st[t0 + kMtHalf];
            uint32_t a1 = mt_mix(hi, st[t0 + kMtHalf + 1]);
            if (has) {
                a[t] = a0;
                a[t + kMtHalf] = a1;
            }
            role_sync(2);
            if (t == kMtHalf - 1) a1 = mt_mix(hi, a[0]);  // word 623 mixes with the new word 0
            a0 ^= a[t0 - 227];
            a1 ^= a[t0 + kMtHalf - 227] ^ a[t0 + kMtHalf - 454];
            if (has) {
                st[t] = a0;
                st[t + kMtHalf] = a1;
            }
            role_sync(2);
            if (has) {
                out[t] = mt_temper(a0);
                out[t + kMtHalf] = mt_temper(a1);
            }
        }
    };
    if (!draws) {
        refill(words[0]);
        for (int buf = 1;; buf ^= 1) {
            __syncthreads();  // words[buf ^ 1] are there, words[buf] used up
            if (stop[buf ^ 1] != 0) return;
            refill(words[buf]);
        }
    }
    int32_t* lst = last + static_cast<size_t>(r) * keep;
    int32_t* hd = head + static_cast<size_t>(r) * keep;
    int32_t* ct = cnt + static_cast<size_t>(r) * (keep + 1);
    const uint32_t K = static_cast<uint32_t>(keep);
    uint32_t i = 1;  // the next draw
    int slot = 0;
    uint32_t refills_left = 2 * (m / kDrawWords) + 16;
    for (int buf = 0;; buf ^= 1) {
        __syncthreads();
        if (stop[buf] != 0) return;
        uint32_t w[2 * kDrawBlocks];
#pragma unroll
        for (int q = 0; q < 2 * kDrawBlocks; ++q) w[q] = words[buf][t0 + q * kMtHalf];
        for (int pos = 0; pos < kDrawWords && i < m;) {  // words before pos are settled
            const uint32_t off = has ? static_cast<uint32_t>(t0 - pos) : 0x80000000u;
            const uint32_t left = static_cast<uint32_t>(kDrawWords - pos);
            unsigned near = 0;
#pragma unroll
            for (int q = 0; q < 2 * kDrawBlocks; ++q) {
                const uint32_t o = off + q * kMtHalf, d = i + o;
                if (w[q] * (d + 1u) <= d && o < left) near |= 1u << q;
            }
            for (; near != 0; near &= near - 1) {
                const uint32_t o = off + (__ffs(near) - 1) * kMtHalf, range = i + o + 1u;
                const uint32_t low = words[buf][pos + o] * range;
                if (low < (0u - range) % range) {
                    atomicMin(&first[slot], pos + static_cast<int>(o));
                    break;
                }
            }
            role_sync(1);
            const int f = first[slot];
            if (t == 0) first[slot == 0 ? 2 : slot - 1] = kDrawWords;
            slot = slot == 2 ? 0 : slot + 1;
            const uint32_t span = min(static_cast<uint32_t>(f - pos), m - i);  // draws settled
#pragma unroll
            for (int q = 0; q < 2 * kDrawBlocks; ++q) {
                const uint32_t o = off + q * kMtHalf, d = i + o, j = __umulhi(w[q], d + 1u);
                asm volatile(
                    "{\n .reg .pred p;\n setp.ne.u32 p, %0, 0;\n @p red.global.max.s32 [%1], %2;\n}" ::"r"(
                        static_cast<uint32_t>(j < K && o < span)),
                    "l"(lst + j), "r"(d)
                    : "memory");
            }
            if (i < K) {  // some are draws of the prefix itself
#pragma unroll
                for (int q = 0; q < 2 * kDrawBlocks; ++q) {
                    const uint32_t o = off + q * kMtHalf, d = i + o, j = __umulhi(w[q], d + 1u);
                    if (j < K && o < span && d < K) {
                        hd[d] = static_cast<int32_t>(j);
                        atomicAdd(ct + j, 1);
                    }
                }
            }
            i += static_cast<uint32_t>(f - pos);
            pos = f + 1;  // a rejected word is consumed; its draw takes the next word
        }
        if (t == 0 && (i >= m || refills_left == 0)) {
            if (i < m) atomicExch(err, 1);
            stop[buf ^ 1] = 1;
        }
        --refills_left;
    }
}

// cnt[r][0..keep) -> inclusive prefix sums (bucket ends); cnt[r][keep] = keep - 1 draws.
__global__ void __launch_bounds__(kScanThreads)
    shuffle_scan_kernel(const long long* __restrict__ ms, int keep, int32_t* __restrict__ cnt) {
    using Scan = cub::BlockScan<int, kScanThreads>;
    __shared__ typename Scan::TempStorage tmp;
    const int r = blockIdx.x;
    if (ms[r] < 2) return;
    int32_t* ct = cnt + static_cast<size_t>(r) * (keep + 1);
    int carry = 0;
    for (int base = 0; base < keep; base += kScanThreads * kScanItems) {
        int v[kScanItems];
        const int i0 = base + threadIdx.x * kScanItems;
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) v[k] = i0 + k < keep ? ct[i0 + k] : 0;
        int total;
        Scan(tmp).InclusiveSum(v, v, total);
#pragma unroll
        for (int k = 0; k < kScanItems; ++k)
            if (i0 + k < keep) ct[i0 + k] = v[k] + carry;
        carry += total;
        __syncthreads();  // tmp is reused by the next tile
    }
    if (threadIdx.x == 0) ct[keep] = keep - 1;
}

// Head step t (1 <= t < keep) goes into bucket head[t]; afterwards cnt[q] is the start of
// bucket q and cnt[q + 1] its end.
__global__ void shuffle_bucket_kernel(const long long* __restrict__ ms, int keep, const int32_t* __restrict__ head,
                                      int32_t* __restrict__ cnt, int32_t* __restrict__ items) {
    const int r = blockIdx.y;
    if (ms[r] < 2) return;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < 1 || t >= keep) return;
    const size_t o = static_cast<size_t>(r) * keep;
    const int q = head[o + t];
    if (q < 0 || q >= keep) return;  // only after a draw run that stopped early (reported by *err)
    const int at = atomicSub(cnt + static_cast<size_t>(r) * (keep + 1) + q, 1) - 1;
    if (at >= 0 && at < keep - 1) items[o + at] = t;
}

// Slot p: last[p] when a step wrote it, else the walk over earlier slots.
__global__ void shuffle_resolve_kernel(const long long* __restrict__ ms, int keep, int32_t* __restrict__ last,
                                       const int32_t* __restrict__ head, const int32_t* __restrict__ cnt,
                                       const int32_t* __restrict__ items) {
    const int r = blockIdx.y;
    if (ms[r] < 1) return;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= keep) return;
    const size_t o = static_cast<size_t>(r) * keep;
    int32_t* lst = last + o;
    if (lst[p] >= 0) return;
    if (p == 0) {  // slot 0 starts as 0 (a range with ms[r] == 1 has only this slot)
        lst[0] = 0;
        return;
    }
    const int32_t* hd = head + o;
    const int32_t* ct = cnt + static_cast<size_t>(r) * (keep + 1);
    const int32_t* it = items + o;
    int q = hd[p];
    int s = p - 1;
    int out = 0;
    // q falls at every step; the index checks only matter after a draw run that stopped
    // early (reported by *err), when head and cnt are incomplete
    for (int guard = 0; guard <= keep && q >= 0 && q < keep; ++guard) {
        int best = -1;
        const int k1 = min(ct[q + 1], keep - 1);
        for (int k = max(ct[q], 0); k < k1; ++k) {
            const int v = it[k];
            if (v <= s && v > best) best = v;
        }
        if (best >= 0) {
            out = best;
            break;
        }
        if (q == 0) break;  // slot 0 starts as 0
        s = q - 1;
        q = hd[q];
    }
    lst[p] = out;
}

}  // namespace

void launch_shuffle_prefix(const uint32_t* seeds, const long long* ms, int n_ranges, int keep, int32_t* out,
                           int32_t* head, int32_t* cnt, int32_t* items, int* err, cudaStream_t s) {
    if (n_ranges <= 0 || keep <= 0) return;
    check(cudaMemsetAsync(out, 0xff, sizeof(int32_t) * static_cast<size_t>(n_ranges) * keep, s), "slots reset");
    check(cudaMemsetAsync(cnt, 0, sizeof(int32_t) * static_cast<size_t>(n_ranges) * (keep + 1), s), "counts reset");
    shuffle_draw_kernel<<<n_ranges, kDrawThreads, 0, s>>>(seeds, ms, keep, out, head, cnt, err);
    check(cudaGetLastError(), "shuffle_draw launch");
    shuffle_scan_kernel<<<n_ranges, kScanThreads, 0, s>>>(ms, keep, cnt);
    check(cudaGetLastError(), "shuffle_scan launch");
    const dim3 grid((keep + 255) / 256, n_ranges);
    shuffle_bucket_kernel<<<grid, 256, 0, s>>>(ms, keep, head, cnt, items);
    check(cudaGetLastError(), "shuffle_bucket launch");
    shuffle_resolve_kernel<<<grid, 256, 0, s>>>(ms, keep, out, head, cnt, items);
    check(cudaGetLastError(), "shuffle_resolve launch");
}

}  // namespace tgb
