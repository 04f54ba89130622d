// Loops of the host's symbolic analysis and partition on a few threads.
#pragma once

#include <algorithm>
#include <atomic>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

namespace mfem {

constexpr int kMaxThreads = 8;

// Runs fn(i) for i in [0, count) on up to `threads` threads, this one
// included; an exception of fn leaves here, as from a plain loop.
template <class F>
inline void parallel_for(int count, int threads, const F &fn) {
    std::atomic<int> next{0};
    std::exception_ptr failed;
    std::mutex lock;
    auto work = [&] {
        try {
            for (int i = next++; i < count; i = next++) fn(i);
        } catch (...) {
            std::lock_guard<std::mutex> hold(lock);
            failed = std::current_exception();
            next = count;
        }
    };
    std::vector<std::thread> pool;
    pool.reserve(std::max(0, std::min(threads, count) - 1));
    try {
        for (int t = 1; t < std::min(threads, count); ++t) pool.emplace_back(work);
    } catch (...) {  // no more threads, or no memory for one: the ones there are do it
    }
    work();
    for (auto &t : pool) t.join();
    if (failed) std::rethrow_exception(failed);
}

// A thread for every `each` rows: enough work to outweigh its start (some 20 us).
inline int thread_count(int rows, int each) {
    const int hw = (int)std::thread::hardware_concurrency();
    return std::max(1, std::min(std::min(kMaxThreads, hw), rows / each));
}

// Rows [0, n) in equal blocks, one a thread: fn(block, first, last).
template <class F>
inline void parallel_rows(int n, int threads, const F &fn) {
    parallel_for(threads, threads, [&](int i) {
        fn(i, (int)((int64_t)n * i / threads), (int)((int64_t)n * (i + 1) / threads));
    });
}

}  // namespace mfem
