// host_threads.h — a parallel loop on the host's threads; set-up done once per device.
#pragma once
#include <algorithm>
#include <atomic>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

// f(0) ... f(n - 1) on the host's threads, the calling one among them, a thread
// for every per_thread of them.  Where fewer threads can be had, those do the
// work; an exception of f ends the loop and is the caller's.
template <class F>
void parallel_for(int n, int per_thread, F&& f)
{
    const int nt = std::max(1, std::min(n / per_thread, (int)std::thread::hardware_concurrency()));
    std::atomic<int> next{0};
    std::mutex mu;
    std::exception_ptr failed;
    auto work = [&] {
        try {
            for (int i = next++; i < n; i = next++) f(i);
        } catch (...) {
            std::lock_guard<std::mutex> lock(mu);
            if (!failed) failed = std::current_exception();
            next = n;
        }
    };
    std::vector<std::thread> others;
    others.reserve((size_t)nt - 1);
    try {
        for (int t = 1; t < nt; t++) others.emplace_back(work);
    } catch (const std::exception&) {                     // no more threads
    }
    work();
    for (auto& t : others) t.join();
    if (failed) std::rethrow_exception(failed);
}

// f() once for each index (a device): a caller that finds it begun by another
// thread waits until it is done.
class OnceEach {
  public:
    template <class F>
    void run(int i, F&& f)
    {
        if (i < 0 || i >= kMost) f();
        else std::call_once(once_[i], f);
    }

  private:
    static constexpr int kMost = 64;
    std::once_flag once_[kMost];
};
