// Host threads of a scene build. One budget is shared by everything that
// builds at the same time, so that a build asked to use N threads never runs
// more than N, the caller's included.
#pragma once

#include <atomic>
#include <future>
#include <system_error>
#include <thread>
#include <type_traits>
#include <utility>
#include <vector>

namespace pray_gpu {

class Threads {
    const int total_;
    std::atomic<int> free_;

  public:
    // total <= 0: every hardware thread
    explicit Threads(int total) : total_(total > 0 ? total : hardware()), free_(total_ - 1) {}
    int total() const { return total_; }
    static int hardware() {
        const unsigned h = std::thread::hardware_concurrency();
        return h ? (int)h : 1;
    }

    // Runs f on a thread of its own if the budget and the system have one;
    // else returns an empty future and the caller does the work itself. What f
    // throws comes out of get(), and a future that goes out of scope waits for
    // its thread, so no exception on either side ends the process.
    template <class F>
    std::future<std::invoke_result_t<F>> start(F f) {
        int n = free_.load();
        do {
            if (n <= 0) return {};
        } while (!free_.compare_exchange_weak(n, n - 1));
        struct Give {
            Threads &t;
            ~Give() { t.free_++; }
        };
        try {
            return std::async(std::launch::async, [this, f = std::move(f)]() mutable {
                Give give{*this};
                return f();
            });
        } catch (const std::system_error &) {  // no more threads to be had
            free_++;
            return {};
        } catch (...) {
            free_++;
            throw;
        }
    }

    // f(0) ... f(count - 1), on the caller and on as many threads as there are.
    template <class F>
    void each(int count, F f) {
        std::atomic<int> next{0};
        auto work = [&] {
            for (int i; (i = next++) < count;) f(i);
        };
        std::vector<std::future<void>> others;
        for (int i = 1; i < count; i++) {
            auto other = start(work);
            if (!other.valid()) break;
            others.push_back(std::move(other));
        }
        work();
        for (auto &o : others) o.get();
    }
};

}  // namespace pray_gpu
