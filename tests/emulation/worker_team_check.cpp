// A team of threads where memory runs out while they are started.
#include "device/worker_team.hpp"

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>

namespace {
std::atomic<int> allocations_left { -1 }; // < 0: no limit
}

void* operator new(std::size_t n)
{
    if (allocations_left.load() >= 0 && allocations_left.fetch_sub(1) <= 0) {
        allocations_left = 0;
        throw std::bad_alloc();
    }
    if (void* p = std::malloc(n))
        return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

int main()
{
    int wrong = 0;
    for (int limit = -1; limit < 12; ++limit) {
        std::atomic<int> next { 0 }, done { 0 };
        allocations_left = limit;
        dxmc_gb300::run_team(8, [&](int) {
            while (next.fetch_add(1) < 1000)
                ++done;
        });
        allocations_left = -1;
        wrong += done != 1000;
    }
    std::printf("runs with pieces left: %d\n", wrong);
    return wrong ? 1 : 0;
}
