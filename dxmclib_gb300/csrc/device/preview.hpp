// Which copies of a job's tally a preview reads while the job may be running.
#pragma once

#include <cstdint>

namespace dxmc_gb300 {

// A job whose transport kernel adds to `copies` of its tally adds copies 1, 2, ... to copy 0
// in a kernel of its own before it ends.  ended(): the job has ended; swept(): its transport
// kernel has, so that the copies may be being added up; wait(): returns once the job has ended;
// read(n): the sum over the first n copies.  A sum over all copies counts some voxels twice if
// they were being added up meanwhile: then copy 0 is read again, once it is complete.
template <class Ended, class Swept, class Wait, class Read>
auto read_tally(std::uint32_t copies, Ended&& ended, Swept&& swept, Wait&& wait, Read&& read) -> decltype(read(copies))
{
    if (copies == 1 || ended())
        return read(1u);
    if (!swept()) {
        const auto result = read(copies);
        if (result || !swept()) // failed, or nothing was added to copy 0 before the read was over
            return result;
    }
    if (const auto failed = wait())
        return failed;
    return read(1u);
}

} // namespace dxmc_gb300
