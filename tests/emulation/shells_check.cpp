// Partial sums over a material's shells against sums in the kernel's own precision.
#include "kernels/shells.hpp"

#include <cstdint>
#include <cstdio>
#include <cstring>
#include <initializer_list>

using namespace dxmc_gb300::dev;

namespace {

// the sums as the kernels' rule states them: every shell bound below E, in order, in Real
template <int WHICH, class Real>
int differ(const float* shells, const float* ready, Real E)
{
    Real cum[N_SHELLS], expected[N_SHELLS], total = 0;
    for (int s = 0; s < N_SHELLS; ++s) {
        const float* sh = shells + s * SHELL_FLOATS;
        const Real weight = WHICH == 0 ? (sh[2] > 0.0f ? sh[1] : 0.0f) : sh[3];
        total += Real(sh[0]) < E ? weight : Real(0);
        expected[s] = total;
    }
    shell_sums<WHICH>(shells, ready, E, cum);
    return std::memcmp(cum, expected, sizeof(cum)) != 0;
}

} // namespace

int main()
{
    std::uint64_t state = 1;
    const auto random = [&state] { return static_cast<float>(dxmc_gb300::splitmix64(state) >> 40) * 0x1p-24f; };
    int wrong32 = 0, wrong64 = 0;
    for (int material = 0; material < 2000; ++material) {
        float shells[N_SHELLS * SHELL_FLOATS] = {}, sums[SHELL_SUM_FLOATS] = {};
        const int present = 1 + material % N_SHELLS;
        for (int s = 0; s < present; ++s) {
            float* sh = shells + s * SHELL_FLOATS;
            sh[0] = 90.0f * random();             // binding energy (keV)
            sh[1] = 10.0f * random();             // electrons
            sh[2] = s % 5 == 4 ? 0.0f : random(); // Compton profile
            sh[3] = random();                     // photoelectric share
        }
        fill_shell_sums(shells, sums);
        for (const float E : { 1.0f, 30.0f, 60.0f, shells[0], sums[2 * N_SHELLS], 100.0f, 150.0f }) {
            wrong32 += differ<0, float>(shells, sums, E) + differ<1, float>(shells, sums, E);
            wrong64 += differ<0, double>(shells, sums, E) + differ<1, double>(shells, sums, E);
        }
    }
    std::printf("lists that differ: %d in FP32, %d in FP64\n", wrong32, wrong64);
    return wrong32 || wrong64 ? 1 : 0;
}
