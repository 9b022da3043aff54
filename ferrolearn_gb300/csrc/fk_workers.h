// fk_workers.h -- a few host threads for one piece of work (host code only).
#pragma once

#include <functional>
#include <thread>

namespace fk {

// work(w) for every w in [0, n), n <= MAX: 0 by the caller, each of the others by a
// thread of its own, or by the caller where none can be had (no thread, or no
// memory for one). All have returned when this does. Nothing is thrown, and
// work must not throw.
template <int MAX, typename Work>
void run_workers(int n, Work &&work) noexcept {
    std::thread pool[MAX];
    bool here[MAX] = {};
    for (int w = 1; w < n; w++) {
        try {
            pool[w] = std::thread(std::ref(work), w);
        } catch (...) {
            here[w] = true;
        }
    }
    if (n > 0) work(0);
    for (int w = 1; w < n; w++)
        if (here[w]) work(w);
    for (int w = 1; w < n; w++)
        if (pool[w].joinable()) pool[w].join();
}

}  // namespace fk
