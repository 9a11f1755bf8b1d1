// Host work on several threads (no CUDA headers, so that it can be checked on its own).
#pragma once

#include <thread>
#include <vector>

namespace omv {

// Runs worker() on up to `threads` threads, the calling one among them, and
// returns when all are done.  A thread that cannot be started (no thread or no
// memory to be had) is left out: the others do its work.  worker() must not throw.
template <typename Worker>
void on_threads(unsigned threads, Worker&& worker)
{
    std::vector<std::thread> pool;
    try {
        pool.reserve(threads);
        for (unsigned k = 1; k < threads; ++k) pool.emplace_back([&worker] { worker(); });
    } catch (...) {
    }
    worker();
    for (std::thread& t : pool) t.join();
}

}  // namespace omv
