// for_each_on_cores when the k-th allocation of the calling thread fails, for k from 0 on: every item is
// done once, or std::bad_alloc comes out. argv[1]: the items.
#include "host_threads.h"

#include <cstdio>
#include <cstdlib>
#include <new>

static thread_local long g_left = -1; // allocations until one fails; -1: none does

void *operator new(size_t n) {
    if (g_left >= 0 && g_left-- == 0)
        throw std::bad_alloc();
    if (void *p = std::malloc(n ? n : 1))
        return p;
    throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }

int main(int argc, char **argv) {
    const uint32_t n = argc > 1 ? static_cast<uint32_t>(std::atoi(argv[1])) : 64;
    for (long k = 0; k < 40; k++) {
        std::vector<uint32_t> order(n);
        std::vector<std::atomic<int>> done(n);
        for (uint32_t i = 0; i < n; i++)
            order[i] = n - 1 - i;
        bool refused = false;
        g_left = k;
        try {
            e8g::for_each_on_cores(order, [&](uint32_t i) { done[i]++; });
        } catch (std::bad_alloc const &) {
            refused = true;
        }
        g_left = -1;
        for (uint32_t i = 0; i < n && !refused; i++)
            if (done[i] != 1)
                return std::printf("allocation %ld: item %u done %d times\n", k, i, done[i].load()), 1;
    }
    bool thrown = false;
    try { // an exception of a call comes out, whichever thread ran it
        e8g::for_each_on_cores(std::vector<uint32_t>(n, 7), [](uint32_t i) { throw i; });
    } catch (uint32_t i) {
        thrown = i == 7;
    }
    return thrown || n == 0 ? 0 : 2;
}
