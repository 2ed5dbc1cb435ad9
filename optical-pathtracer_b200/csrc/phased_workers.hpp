// Host threads that work in two phases, the second starting when all of them are done with the first.
#pragma once

#include <atomic>
#include <exception>
#include <functional>
#include <limits>
#include <mutex>
#include <thread>
#include <vector>

namespace owec {

// run(first, second): first(worker) on every worker, and once all of them are done with it second(worker) on every
// worker. The calling thread is worker 0; the others are started here, as many as the system gives
// (with none, the calling thread does all the work, which the callers deal out piece by piece). After a failure
// no further phase starts; the first one is rethrown once all threads have ended. Thread: std::thread, or a
// test's.
template <class Thread = std::thread>
class PhasedWorkersOf {
public:
    explicit PhasedWorkersOf(int workers) : wanted_(workers) {}

    void run(const std::function<void(int)>& first, const std::function<void(int)>& second) {
        threads_.reserve(size_t(wanted_));
        for (int k = 1; k < wanted_; ++k) {
            try {
                threads_.emplace_back([this, k, &first, &second] {
                    attempt([&] { first(k); });
                    waitForAll();
                    attempt([&] { second(k); });
                });
            } catch (...) {  // no more threads to be had
                break;
            }
        }
        expected_ = int(threads_.size()) + 1;
        attempt([&] { first(0); });
        waitForAll();
        attempt([&] { second(0); });
        for (Thread& t : threads_) t.join();
        if (failure_) std::rethrow_exception(failure_);
    }

private:
    // The phases' ends lie microseconds apart, less than waking a sleeping thread takes.
    void waitForAll() {
        ++arrived_;
        while (arrived_ < expected_) std::this_thread::yield();
    }

    // f(), unless something has failed before.
    void attempt(const std::function<void()>& f) {
        {
            std::lock_guard<std::mutex> lock(mutex_);
            if (failure_) return;
        }
        try {
            f();
        } catch (...) {
            std::lock_guard<std::mutex> lock(mutex_);
            if (!failure_) failure_ = std::current_exception();
        }
    }

    int wanted_;
    std::atomic<int> arrived_{0}, expected_{std::numeric_limits<int>::max()};
    std::mutex mutex_;
    std::exception_ptr failure_;
    std::vector<Thread> threads_;
};
using PhasedWorkers = PhasedWorkersOf<>;

}  // namespace owec
