// How the warps of a transport kernel share a job's histories (or queued photons),
// usable from host and device code: the host runs the warp's side of it in a test that
// lets the lanes advance one at a time.
#pragma once

#include "stream_seed.hpp" // DXMC_HD

#include <cstdint>

namespace dxmc_gb300 {

// A job's ids in units that a warp takes at a time: `large_units` of `large` ids, then
// units of `small` (both multiples of 32).
struct WorkSplit {
    std::uint64_t large_units = 0;
    std::uint32_t large = 256;
    std::uint32_t small = 32;
};

// Threads of a block for a wish of the caller's: whole warps.  A kernel whose last warp has
// fewer lanes would give that warp the units of the next block's first, and wait for idle
// lanes that it does not have.
inline int whole_warps(int threads) { return threads > 32 ? (threads + 31) / 32 * 32 : 32; }

// The ids of one unit of a job's work; a unit past the end starts at or after the job's
// last id.
DXMC_HD inline std::uint64_t work_unit(const WorkSplit& w, std::uint64_t unit, std::uint64_t& end)
{
    const bool large = unit < w.large_units;
    const std::uint64_t first = large ? unit * w.large : w.large_units * w.large + (unit - w.large_units) * w.small;
    end = first + (large ? w.large : w.small);
    return first;
}

// The ids handed out once the queue has given `fetched` units beside the first ones of
// `warps` warps.
inline std::uint64_t ids_taken(const WorkSplit& w, std::uint64_t warps, std::uint64_t fetched, std::uint64_t total)
{
    std::uint64_t end;
    const std::uint64_t first = work_unit(w, warps + fetched, end);
    return first < total ? first : total;
}

// In the queue's counter: the job was cancelled, its units go to nobody any more.  The
// count below it stays what it is.
constexpr std::uint64_t QUEUE_STOPPED = 1ull << 63;
// Units between two looks at the host's cancel flag, which costs a read over the link (a
// microsecond); the warp that finds it set stops the queue for all.  A block looks once
// before its first units, so a job cancelled while it waits does no work.
constexpr std::uint64_t CANCEL_CHECK_UNITS = 32;

// The first of the ids that a warp samples next: the rest of its unit, or a new unit,
// the queue's next one after the first `warps`; `total` or more once there is none.
// `ids` (next, end) is the warp's shared state.  Called by all lanes of the warp, which get
// the same value; the caller advances ids.next.  Warp: leader(), sync(), broadcast(value of
// the leader), fetch_add(address), stop(address).
template <class Warp, class Ids, class Cancelled>
DXMC_HD inline std::uint64_t next_ids(Warp& warp, Ids& ids, const WorkSplit& work, std::uint64_t warps, unsigned long long* head,
    std::uint64_t total, Cancelled&& cancelled)
{
    std::uint64_t next = ids.next;
    if (next >= ids.end) {
        // every lane has read ids.end before the leader writes it
        warp.sync();
        if (warp.leader()) {
            const std::uint64_t fetched = warp.fetch_add(head);
            const std::uint64_t unit = warps + fetched;
            std::uint64_t end;
            next = work_unit(work, unit, end);
            ids.end = end;
            if (fetched & QUEUE_STOPPED) {
                next = total;
            } else if (unit % CANCEL_CHECK_UNITS == 0 && cancelled()) {
                warp.stop(head);
                next = total;
            }
        }
        next = warp.broadcast(next);
    }
    return next;
}

} // namespace dxmc_gb300
