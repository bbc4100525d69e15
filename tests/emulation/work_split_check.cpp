// A warp's way through a job's work units (next_ids), with lanes that advance one at a time.
#include "kernels/work_split.hpp"
#include "warp_lanes.hpp"

#include <algorithm>
#include <initializer_list>

using namespace dxmc_gb300;

namespace {

struct Ids {
    std::uint64_t next = 0, end = 0;
};

int failures = 0;
void check(bool ok, const char* what)
{
    if (!ok) {
        std::printf("FAIL %s\n", what);
        ++failures;
    }
}

// What the progress says after each unit that the queue gives: the ids handed out, up to the
// job's total.
void progress_counts_ids(const WorkSplit& work, std::uint64_t warps, std::uint64_t total)
{
    std::uint64_t end, handed = 0;
    bool same = true;
    for (std::uint64_t unit = 0;; ++unit) {
        if (unit >= warps)
            same = same && ids_taken(work, warps, unit - warps, total) == std::min(handed, total);
        const std::uint64_t first = work_unit(work, unit, end);
        handed += end - first;
        if (unit > warps && first >= total)
            break;
    }
    check(same, "the progress is the number of ids handed out");
}

// One warp takes all units of a job of `total` ids: every id once, all lanes the same.
void all_ids_once(const WorkSplit& work, std::uint64_t total, bool ascending)
{
    Ids ids;
    ids.next = work_unit(work, 0, ids.end);
    unsigned long long head = 0;
    std::vector<int> taken(total, 0);
    emulation::Warp warp;
    const bool converged = warp.run(
        [&](emulation::Warp& w, int lane) {
            while (true) {
                const std::uint64_t next = next_ids(w, ids, work, 1, &head, total, [] { return false; });
                if (next >= total)
                    break;
                if (next + lane < total)
                    ++taken[next + lane];
                w.sync(); // the votes over the sampled photons
                if (w.leader())
                    ids.next = next + 32;
                w.sync();
            }
        },
        ascending);
    check(converged, "lanes meet at the same collective");
    check(std::all_of(taken.begin(), taken.end(), [](int n) { return n == 1; }), "every id is taken once");
}

// The flag is set once `set_after` ids have been handed out; what the queue gives after that,
// to this warp and to another one that never looks at the flag itself.
void stops_when_cancelled(const WorkSplit& work, std::uint64_t total, std::uint64_t set_after)
{
    Ids ids;
    ids.next = work_unit(work, 0, ids.end);
    unsigned long long head = 0;
    std::uint64_t taken = 0;
    emulation::Warp warp;
    warp.run(
        [&](emulation::Warp& w, int) {
            while (true) {
                const std::uint64_t next = next_ids(w, ids, work, 1, &head, total, [&] { return taken >= set_after; });
                if (next >= total)
                    break;
                w.sync();
                if (w.leader()) {
                    ids.next = next + 32;
                    taken += 32;
                }
                w.sync();
            }
        },
        true);
    check(taken < set_after + CANCEL_CHECK_UNITS * std::max(work.large, work.small) + 32, "the flag is seen within a few units");
    Ids other;
    bool stopped = false;
    warp.run([&](emulation::Warp& w, int) { stopped = next_ids(w, other, work, 1, &head, total, [] { return false; }) >= total; }, true);
    check(stopped, "the queue is stopped for the other warps");
}

} // namespace

int main()
{
    for (const std::uint64_t warps : { 1u, 7u, 64u })
        for (const std::uint64_t total : { 1u, 100u, 5000u, 100000u }) {
            WorkSplit work;
            progress_counts_ids(work, warps, total);
            work.large = 96;
            work.large_units = std::min<std::uint64_t>(warps, total / work.large);
            progress_counts_ids(work, warps, total);
            work.large_units = total / work.large / 2;
            work.small = 64;
            progress_counts_ids(work, warps, total);
        }
    for (int threads = 1; threads <= 256; ++threads) {
        const int block = whole_warps(threads);
        check(block % 32 == 0 && block >= threads && block < threads + 32, "a block is whole warps");
    }
    WorkSplit split;
    stops_when_cancelled(split, 1u << 20, 0); // small units only
    stops_when_cancelled(split, 1u << 20, 5000);
    split.large_units = 1; // as in jobs of a few rounds: the queue hands out small ones only
    stops_when_cancelled(split, 1u << 20, 5000);
    split.large_units = 200; // cancelled among the last, small units
    stops_when_cancelled(split, 1u << 20, 200 * 256 + 1000);
    for (const bool ascending : { true, false })
        for (const std::uint64_t total : { 1u, 31u, 32u, 33u, 700u, 1500u }) {
            WorkSplit work; // small units only
            all_ids_once(work, total, ascending);
            work.large_units = 2; // two large units, then small ones
            all_ids_once(work, total, ascending);
            work.small = 64;
            all_ids_once(work, total, ascending);
        }
    std::printf(failures ? "%d checks failed\n" : "ok\n", failures);
    return failures ? 1 : 0;
}
