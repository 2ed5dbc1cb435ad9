// Host threads that work in two phases, the second starting when all of them are done with the first.
#pragma once

#include <condition_variable>
#include <exception>
#include <functional>
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
                    {
                        std::unique_lock<std::mutex> lock(mutex_);
                        ++arrived_;
                        changed_.notify_all();
                        changed_.wait(lock, [&] { return open_; });
                    }
                    attempt([&] { second(k); });
                });
            } catch (...) {  // no more threads to be had
                break;
            }
        }
        attempt([&] { first(0); });
        {
            std::unique_lock<std::mutex> lock(mutex_);
            changed_.wait(lock, [&] { return arrived_ == int(threads_.size()); });
            open_ = true;
            changed_.notify_all();
        }
        attempt([&] { second(0); });
        for (Thread& t : threads_) t.join();
        if (failure_) std::rethrow_exception(failure_);
    }

private:
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

    int wanted_, arrived_ = 0;
    bool open_ = false;
    std::mutex mutex_;
    std::condition_variable changed_;
    std::exception_ptr failure_;
    std::vector<Thread> threads_;
};
using PhasedWorkers = PhasedWorkersOf<>;

}  // namespace owec
