// A preview beside the kernel that adds up the copies of a tally: every timing of the two.
#include "device/preview.hpp"

#include <cstdio>
#include <vector>

namespace {

constexpr int VOXELS = 8;
constexpr unsigned COPIES = 4;

// Time passes with every query and with every voxel read; the copies are added up from tick
// `start` to tick `end`, some blocks at once and the others, which wait for an SM, at the end.
struct Timeline {
    int start, end, now = 0;
    double at(unsigned copy, int voxel) const
    {
        const double own = 1.0 + copy + 10.0 * voxel;
        if (copy > 0)
            return own;
        const int when = voxel % 2 ? end : start;
        double sum = own;
        for (unsigned c = 1; now >= when && c < COPIES; ++c)
            sum += 1.0 + c + 10.0 * voxel;
        return sum;
    }
};

} // namespace

int main()
{
    int wrong = 0, waits = 0;
    for (int start = 0; start < 120; ++start)
        for (int length = 0; length < 60; ++length) {
            Timeline t { start, start + length };
            std::vector<double> energy(VOXELS);
            const int failed = dxmc_gb300::read_tally(
                COPIES, [&] { return t.now++ >= t.end; }, [&] { return t.now++ >= t.start; },
                [&] {
                    t.now = t.now > t.end ? t.now : t.end;
                    ++waits;
                    return 0;
                },
                [&](unsigned copies) {
                    for (unsigned c = 0; c < copies; ++c)
                        for (int v = 0; v < VOXELS; ++v, ++t.now)
                            energy[v] = c == 0 ? t.at(0, v) : energy[v] + t.at(c, v);
                    return 0;
                });
            bool right = !failed;
            for (int v = 0; v < VOXELS; ++v)
                right = right && energy[v] == 10.0 + 40.0 * v;
            wrong += !right;
        }
    std::printf("wrong previews: %d; waits for the end: %d\n", wrong, waits);
    return wrong || !waits ? 1 : 0;
}
