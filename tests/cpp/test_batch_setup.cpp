// Host-only checks of the batched fits' set-ups (tidegbm_b200/csrc/batch_setup.h) on a device that is
// a counter: a set-up holds its upload while it runs and its context from then on.  Built and run by
// tests/test_cpu_batch_setup.py; prints "ok".
#include "batch_setup.h"

#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <stdexcept>
#include <string>

#define CHECK(c)                                                        \
    do {                                                                \
        if (!(c)) {                                                     \
            std::fprintf(stderr, "%s:%d: check failed: %s\n", __FILE__, __LINE__, #c); \
            std::exit(1);                                               \
        }                                                               \
    } while (0)

struct Full : std::runtime_error {
    using std::runtime_error::runtime_error;
};

struct Device {
    std::vector<size_t> upload, context;
    size_t capacity, limit;
    int threads = 3;
    int bad = -1;  // a set-up that fails for another reason
    std::mutex mu;
    size_t used = 0, most = 0;
    int running = 0, most_running = 0, undone = 0;
    std::vector<size_t> held;
    std::vector<int> calls;

    Device(std::vector<size_t> u, std::vector<size_t> c, size_t cap, size_t lim = 1000)
        : upload(std::move(u)), context(std::move(c)), capacity(cap), limit(lim), held(upload.size(), 0), calls(upload.size(), 0) {}

    void take(int k, size_t b) {
        std::lock_guard<std::mutex> lk(mu);
        if (used + b > capacity) throw Full("set-up " + std::to_string(k));
        used += b;
        held[k] += b;
        most = std::max(most, used);
    }
    void give(int k, size_t b) {
        std::lock_guard<std::mutex> lk(mu);
        used -= b;
        held[k] -= b;
    }
    void prepare(int k) {
        {
            std::lock_guard<std::mutex> lk(mu);
            ++calls[k];
            most_running = std::max(most_running, ++running);
        }
        struct Done {
            Device& d;
            ~Done() {
                std::lock_guard<std::mutex> lk(d.mu);
                --d.running;
            }
        } done{*this};
        if (k == bad) throw std::invalid_argument("bad " + std::to_string(k));
        take(k, context[k]);
        take(k, upload[k]);  // what was taken stays when this throws, as a booster's buffers do
        std::this_thread::sleep_for(std::chrono::milliseconds(20));
        give(k, upload[k]);
    }
    void undo(int k) {
        ++undone;
        give(k, held[k]);
    }
    void run() {
        tgb::run_setups(
            static_cast<int>(upload.size()), threads, limit, [&](int k) { return upload[k]; }, [&](int k) { prepare(k); },
            [&](int k) { undo(k); },
            [](const std::exception_ptr& e) {
                try {
                    std::rethrow_exception(e);
                } catch (const Full&) {
                    return true;
                } catch (...) {
                    return false;
                }
            });
    }
    std::string error() {
        try {
            run();
        } catch (const std::exception& e) {
            return e.what();
        }
        return "";
    }
};

int main() {
    {  // room for all: side by side, at most three
        Device d({10, 10, 10, 10, 10, 10}, {5, 5, 5, 5, 5, 5}, 1000);
        d.run();
        CHECK(d.most_running == 3 && d.undone == 0 && d.used == 30);
        for (int c : d.calls) CHECK(c == 1);
    }
    {  // uploads beyond the limit take turns
        Device d({60, 60, 30, 30, 200}, {1, 1, 1, 1, 1}, 1000, 100);
        d.run();
        CHECK(d.undone == 0 && d.used == 5 && d.most <= 205);
    }
    {  // no room side by side, room for one after another: every one is set up all the same
        Device d({50, 50, 50, 50}, {10, 10, 10, 10}, 90);
        d.run();
        CHECK(d.undone > 0 && d.used == 40 && d.most <= 90);
        for (size_t h : d.held) CHECK(h == 10);
    }
    {  // the largest first: its contexts' neighbours have to go again before it fits
        Device d({70, 10, 10}, {10, 10, 10}, 85);
        d.run();
        CHECK(d.used == 30);
    }
    {  // no room even alone: the error of the set-up that would have failed in order
        Device d({20, 90, 20}, {10, 10, 10}, 85);
        CHECK(d.error() == "set-up 1");
        CHECK(d.calls[2] <= 1);
    }
    {  // another error is not tried again, and nothing starts behind it
        Device d({10, 10, 10, 10, 10, 10, 10, 10}, {1, 1, 1, 1, 1, 1, 1, 1}, 1000);
        d.bad = 1;
        CHECK(d.error() == "bad 1");
        CHECK(d.undone == 0 && d.calls[1] == 1 && d.calls[7] == 0);
    }
    {  // a set-up without room, then a bad one: in order the bad one is what fails
        Device d({50, 50, 50, 50}, {10, 10, 10, 10}, 90);
        d.bad = 3;
        CHECK(d.error() == "bad 3");
    }
    {  // one thread, one set-up
        Device d({10, 10}, {1, 1}, 12);
        d.threads = 1;
        d.run();
        CHECK(d.most_running == 1 && d.undone == 0);
        Device e({10}, {1}, 5);
        CHECK(e.error() == "set-up 0");
    }
    std::puts("ok");
    return 0;
}
