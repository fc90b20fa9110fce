// Runs the set-ups of a batched fit side by side (GpuBooster::fit_batch).  Host only; checked by
// tests/cpp/test_batch_setup.cpp.
#pragma once

#include <algorithm>
#include <condition_variable>
#include <cstddef>
#include <exception>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace tgb {

// Calls prepare(k) for k = 0 .. n - 1, started in order, at most `threads` at a time and as long as
// the bytes(k) of those under way stay within `limit`; a larger one runs alone.  The first failure
// lets no later one start.  It is rethrown, the one of the lowest k where there are several, as if
// they had run one after another, with one exception: side by side they need more memory than one
// after another, so where out_of_memory(error) holds, that set-up and those behind it are taken
// back (undo(k), in any state) and run again, one by one.
template <typename Bytes, typename Prepare, typename Undo, typename OutOfMemory>
void run_setups(int n, int threads, size_t limit, Bytes bytes, Prepare prepare, Undo undo, OutOfMemory out_of_memory) {
    std::mutex mu;
    std::condition_variable cv;
    int next = 0, running = 0;
    size_t under_way = 0;
    bool stop = false;
    std::vector<std::exception_ptr> failed(n);
    auto work = [&] {
        while (true) {
            int k;
            {
                std::unique_lock<std::mutex> lk(mu);
                cv.wait(lk, [&] { return stop || next >= n || running == 0 || under_way + bytes(next) <= limit; });
                if (stop || next >= n) return;
                k = next++;
                under_way += bytes(k);
                ++running;
            }
            try {
                prepare(k);
            } catch (...) {
                failed[k] = std::current_exception();
            }
            {
                std::lock_guard<std::mutex> lk(mu);
                under_way -= bytes(k);
                --running;
                if (failed[k]) stop = true;
            }
            cv.notify_all();
        }
    };
    {
        struct Joined {  // also where a thread cannot be started, or work() throws
            std::vector<std::thread> th;
            ~Joined() {
                for (auto& t : th) t.join();
            }
        } joined;
        joined.th.reserve(std::max(0, threads - 1));
        for (int t = 1; t < std::min(threads, n); ++t) {
            try {
                joined.th.emplace_back(work);
            } catch (const std::system_error&) {
                break;  // fewer side by side
            }
        }
        work();
    }
    const int first = static_cast<int>(std::find_if(failed.begin(), failed.end(), [](auto& f) { return f != nullptr; }) - failed.begin());
    if (first == n) return;
    if (!out_of_memory(failed[first])) std::rethrow_exception(failed[first]);
    for (int k = first; k < next; ++k) undo(k);
    for (int k = first; k < n; ++k) prepare(k);
}

}  // namespace tgb
