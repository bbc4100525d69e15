// A few host threads for the pieces of one transfer.
#pragma once

#include <exception>
#include <thread>
#include <vector>

namespace dxmc_gb300 {

// Runs work(0) on the calling thread and work(1) .. work(threads - 1) on threads of their own,
// and returns once all have ended.  Where no more threads can be started (their number, or
// memory) those there are take the pieces: work() takes the next one until none is left.
template <class Work>
void run_team(int threads, Work&& work)
{
    std::vector<std::thread> team;
    try {
        team.reserve(static_cast<size_t>(threads));
        for (int t = 1; t < threads; ++t)
            team.emplace_back([&work, t] { work(t); });
    } catch (const std::exception&) { // std::system_error, std::bad_alloc
    }
    work(0);
    for (std::thread& t : team)
        t.join();
}

} // namespace dxmc_gb300
