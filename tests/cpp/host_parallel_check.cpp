// csrc/host_parallel.h when memory runs out: a thread that cannot be made leaves
// its share to the others, an exception of the work reaches the caller with
// every thread joined.  Prints "ok" or what went wrong.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <stdexcept>
#include <vector>

#include "host_parallel.h"

static thread_local int t_until = -1;  // allocations of this thread until one fails; < 0: none does

void *operator new(std::size_t size) {
    if (t_until >= 0 && t_until-- == 0) throw std::bad_alloc();
    if (void *p = std::malloc(size ? size : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, std::size_t) noexcept { std::free(p); }

int main() {
    // the first allocation is the pool's, the further ones a thread each
    for (int until = 1; until <= 4; ++until) {
        std::vector<std::atomic<int>> met(100);
        t_until = until;
        mfem::parallel_for(100, 4, [&](int i) { ++met[i]; });
        t_until = -1;
        for (auto &m : met)
            if (m != 1) {
                puts("an item was lost or repeated");
                return 1;
            }
    }
    std::atomic<int> running{0};
    try {
        mfem::parallel_for(100, 4, [&](int i) {
            ++running;
            const bool bad = i == 37;
            --running;
            if (bad) throw std::runtime_error("item 37");
        });
        puts("the exception was lost");
        return 1;
    } catch (const std::runtime_error &) {
    }
    if (running != 0) return 1;
    puts("ok");
    return 0;
}
