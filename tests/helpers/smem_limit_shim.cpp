// Threads that raise the shared-memory limit of one kernel at the same time (csrc/smem_limit.h), with a stand-in for the
// driver call that takes long enough for them to interleave, the longer the smaller the limit it sets.
#include "smem_limit.h"

#include <chrono>
#include <thread>
#include <vector>

// Number of "launches" that found the limit below what their thread had asked for; calls <- driver calls made.
extern "C" int raise_from_threads(const int* bytes, int n, int* calls) {
    pl::SmemLimit limit;
    std::atomic<int> current{0}, refused{0}, made{0}, waiting{n};
    std::vector<std::thread> threads;
    for (int i = 0; i < n; i++)
        threads.emplace_back([&, want = bytes[i]] {
            waiting--;
            while (waiting > 0) std::this_thread::yield();
            const int rc = limit.raise(0, (size_t)want, [&](size_t b) {
                made++;
                std::this_thread::sleep_for(std::chrono::milliseconds(20 + 2000 / (int)b));
                current = (int)b;
                return 0;
            });
            std::this_thread::sleep_for(std::chrono::milliseconds(100));
            if (rc != 0 || current < want) refused++;
        });
    for (auto& t : threads) t.join();
    *calls = made;
    return refused;
}

// A driver call that fails is reported and tried again by the next caller.
extern "C" int raise_after_failure(void) {
    pl::SmemLimit limit;
    const int first = limit.raise(0, 100, [](size_t) { return 5; });
    int tried = 0;
    const int second = limit.raise(0, 100, [&](size_t) { tried++; return 0; });
    const int third = limit.raise(0, 100, [&](size_t) { tried++; return 0; });
    return first == 5 && second == 0 && third == 0 && tried == 1 ? 0 : 1;
}
