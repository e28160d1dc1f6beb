// dmft-ed-zt_b200/csrc/host_threads.h: set-up done once, before any thread goes
// on; parallel_for where no thread can be had and where the function throws.
// Prints "ok" and returns 0.
#include <chrono>
#include <cstdio>
#include <stdexcept>
#include <vector>
#include <sys/resource.h>
#include <unistd.h>
#include "host_threads.h"

constexpr int n_bad = 0;

static int run(int n)
{
    std::vector<int> hit((size_t)n, 0);
    parallel_for(n, 1, [&](int i) { hit[(size_t)i]++; });
    int bad = 0;
    for (int h : hit) bad += h != 1;
    return bad;
}

// Threads that meet at one index's set-up and see it done.
static int once(int threads)
{
    OnceEach each;
    std::atomic<int> begun{0}, done{0}, early{0};
    std::vector<std::thread> th;
    for (int t = 0; t < threads; t++)
        th.emplace_back([&] {
            each.run(3, [&] {
                begun++;
                std::this_thread::sleep_for(std::chrono::milliseconds(50));
                done++;
            });
            early += done == 0;
        });
    for (auto& t : th) t.join();
    return begun != 1 || done != 1 || early != 0;
}

int main()
{
    if (once(8)) { std::printf("once\n"); return 5; }
    for (int n : {0, 1, 2, 7, 1000})
        if (run(n)) { std::printf("n %d\n", n); return 1; }
    int caught = 0;
    for (int n : {1, 64})
        try {
            parallel_for(n, 1, [](int i) { if (i == n_bad) throw std::runtime_error("f"); });
        } catch (const std::runtime_error&) {
            caught++;
        }
    if (caught != 2) { std::printf("caught %d\n", caught); return 2; }
    // no address space for another thread's stack: std::thread's constructor throws
    unsigned long pages = 0;
    FILE* f = std::fopen("/proc/self/statm", "r");
    if (!f || std::fscanf(f, "%lu", &pages) != 1) return 3;
    std::fclose(f);
    const rlim_t bytes = (rlim_t)pages * (rlim_t)sysconf(_SC_PAGESIZE) + (4u << 20);
    const rlimit lim{bytes, bytes};
    if (setrlimit(RLIMIT_AS, &lim)) return 3;
    if (run(1000)) { std::printf("without threads\n"); return 4; }
    std::printf("ok\n");
    return 0;
}
