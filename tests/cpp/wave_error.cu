// An error noted while one tree grows outlives the set-up of the next, and a later error does not
// replace it (tidegbm_b200/csrc/kernels_wave.cu, kernels_wave_scan.cu).  The overflow is harmless: a
// context whose tile bound is zero, so that the select refuses to plan the root's split and ends the
// tree.  Linked with the library's objects and run by tests/test_gpu_wave_error.py; prints "ok".
#include <cstdio>
#include <cstdlib>

#include "wave.h"

using namespace tgb;

#define CHECK(c)                                                        \
    do {                                                                \
        if (!(c)) {                                                     \
            std::fprintf(stderr, "%s:%d: check failed: %s\n", __FILE__, __LINE__, #c); \
            std::exit(1);                                               \
        }                                                               \
    } while (0)

template <typename T>
static T* zeros(size_t n) {
    void* p = nullptr;
    CHECK(cudaMalloc(&p, n * sizeof(T)) == cudaSuccess);
    CHECK(cudaMemset(p, 0, n * sizeof(T)) == cudaSuccess);
    return static_cast<T*>(p);
}

int main() {
    const int n = 100, n_f = 1;
    const size_t slot = static_cast<size_t>(n_f) * kBins;
    WaveCtx x{};
    x.rows0 = zeros<int32_t>(n);
    x.rows1 = zeros<int32_t>(n);
    x.nodes = zeros<DevNode>(kMaxNodes);
    x.splits = zeros<DevSplit>(kMaxNodes);
    x.st = zeros<DevTreeState>(1);
    x.spec = zeros<DevNode>(2 * kMaxNodes);
    x.spec_split = zeros<DevSplit>(2 * kMaxNodes);
    x.ctl = zeros<WaveCtl>(1);
    x.G = zeros<long long>(slot * 3);
    x.H = zeros<long long>(slot * 3);
    x.C = zeros<int>(slot * 3);
    x.gp = GrowParams{n_f, 16, 255, 4, 4, 1, 0.0, 1.0, 0.0};
    x.n_slots = 3;
    x.max_tiles = 0;  // no room for the root's one tile
    WaveCtx* ctx = zeros<WaveCtx>(1);
    CHECK(cudaMemcpy(ctx, &x, sizeof(x), cudaMemcpyHostToDevice) == cudaSuccess);
    int* gsync = zeros<int>(3);
    AllScale* all = zeros<AllScale>(1);
    unsigned long long* seg = zeros<unsigned long long>(3 * kMaxNodes);
    auto begin = [&] {
        launch_wave_begin(WaveBegin{x.nodes, x.splits, x.st, x.ctl, all, x.G, x.H, x.C, slot, seg, 3 * kMaxNodes, nullptr,
                                    x.rows0, n, 0, kHistExactConst},
                          nullptr);
    };
    auto select = [&] {
        DevSplit s{};
        s.gain = 1.0;
        s.valid = 1;
        CHECK(cudaMemcpy(x.splits, &s, sizeof(s), cudaMemcpyHostToDevice) == cudaSuccess);
        launch_wave_select(ctx, 1, gsync, nullptr, 0ull, 0, nullptr);
    };
    auto error = [&] {
        int e = -1;
        CHECK(cudaMemcpy(&e, &x.ctl->error, sizeof(e), cudaMemcpyDeviceToHost) == cudaSuccess);
        return e;
    };
    begin();
    CHECK(error() == 0);
    select();
    CHECK(error() == 1);
    begin();  // the next tree
    CHECK(error() == 1);
    const int staging = 3;  // a staging wait that gave up, then the overflow
    CHECK(cudaMemcpy(&x.ctl->error, &staging, sizeof(int), cudaMemcpyHostToDevice) == cudaSuccess);
    begin();
    select();
    CHECK(error() == 3);
    std::puts("ok");
    return 0;
}
