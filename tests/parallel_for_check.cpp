// parallel_for (common.hpp) when memory or threads run out while it starts its
// threads: every item is still done once, or the failure comes back as an
// exception; and the exception rethrown is the first in item order.
#include "common.hpp"

#include <cstdio>
#include <cstdlib>
#include <new>

static std::atomic<long> allocations_left{-1};   // -1: no limit

void* operator new(size_t n) {
    if (allocations_left >= 0 && allocations_left.fetch_sub(1) <= 0) {
        allocations_left = 0;
        throw std::bad_alloc();
    }
    if (void* p = std::malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

int main() {
    static std::atomic<int> seen[100000];
    for (long limit = 0; limit < 40; ++limit) {
        for (auto& s : seen) s = 0;
        bool thrown = false;
        allocations_left = limit;
        try {
            fvmb::parallel_for(100000, 1, [&](long a, long b) {
                for (long i = a; i < b; ++i) seen[i]++;
            });
        } catch (const std::bad_alloc&) {
            thrown = true;
        }
        allocations_left = -1;
        for (auto& s : seen)
            if (s > 1 || (s == 0 && !thrown)) {
                std::printf("limit %ld: an item was done %d times\n", limit, (int)s);
                return 1;
            }
    }
    for (int rep = 0; rep < 50; ++rep) {
        long at = -1;
        try {
            fvmb::parallel_for(100000, 1, [&](long a, long b) {
                for (long i = a; i < b; ++i)
                    if (i % 7000 == 6999) throw i;
            });
        } catch (long i) {
            at = i;
        }
        if (at != 6999) {
            std::printf("first failing item %ld\n", at);
            return 1;
        }
    }
    std::printf("ok\n");
    return 0;
}
