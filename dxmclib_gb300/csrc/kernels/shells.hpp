// Choice of the electron shell of a photoelectric or impulse-approximation Compton
// event, usable from host and device code.
#pragma once

#include "stream_seed.hpp" // DXMC_HD

namespace dxmc_gb300::dev {

constexpr int SHELL_FLOATS = 12; // binding, nElectrons, J0, photoProb, yield, lineP[3], lineE[3], pad
constexpr int N_SHELLS = 12;
constexpr int SHELL_SUM_FLOATS = 28; // partial sums over the shells: electrons (J0 > 0)[12], photoProb[12], highest binding energy, pad

// A shell's weight (0: its electrons where it has a Compton profile, 1: photoelectric).
template <int WHICH>
DXMC_HD inline float shell_weight(const float* shell)
{
    return WHICH == 0 ? (shell[2] > 0.0f ? shell[1] : 0.0f) : shell[3];
}

// The shells' partial sums for energies above the material's highest binding energy, where
// every shell takes part: summed in the order and precision of the FP32 kernels, which take
// them ready-made (DX 127^3 with impulse approximation, 4e6 histories: 1.26 -> 1.18 ms).
inline void fill_shell_sums(const float* shells, float* sums)
{
    float electrons = 0.0f, photo = 0.0f, highest = shells[0];
    for (int s = 0; s < N_SHELLS; ++s) {
        const float* sh = shells + s * SHELL_FLOATS;
        sums[s] = electrons += shell_weight<0>(sh);
        sums[N_SHELLS + s] = photo += shell_weight<1>(sh);
        highest = sh[0] > highest ? sh[0] : highest;
    }
    sums[2 * N_SHELLS] = highest;
}

// Partial sums of a material's shells at energy E into cum, in the precision of the caller.
// Kernels in double sum the weights themselves: the LUT's sums are rounded to 24 bits.
template <int WHICH, class Real>
DXMC_HD inline void shell_sums(const float* shells, const float* ready, Real E, Real (&cum)[N_SHELLS])
{
    if constexpr (sizeof(Real) == sizeof(float)) {
        if (E > ready[2 * N_SHELLS]) {
#pragma unroll
            for (int s = 0; s < N_SHELLS; ++s)
                cum[s] = ready[WHICH * N_SHELLS + s];
            return;
        }
        Real total = Real(0.0);
        for (int s = 0; s < N_SHELLS; ++s) { // rolled: seldom taken
            const float* sh = shells + s * SHELL_FLOATS;
            total += sh[0] < E ? shell_weight<WHICH>(sh) : Real(0.0);
#pragma unroll
            for (int k = 0; k < N_SHELLS; ++k) // cum stays in registers
                cum[k] = k == s ? total : cum[k];
        }
    } else {
        Real total = Real(0.0);
#pragma unroll
        for (int s = 0; s < N_SHELLS; ++s) {
            const float* sh = shells + s * SHELL_FLOATS;
            total += Real(sh[0]) < E ? Real(shell_weight<WHICH>(sh)) : Real(0.0);
            cum[s] = total;
        }
    }
}

// The first shell whose partial sum reaches u times the total: the total and the search use
// one list of sums.
template <class Real>
DXMC_HD inline int pick_shell(const Real (&cum)[N_SHELLS], Real u)
{
    const Real sample = cum[N_SHELLS - 1] * u;
    int idx = 0;
#pragma unroll
    for (int s = 0; s < N_SHELLS - 1; ++s)
        idx += cum[s] < sample ? 1 : 0; // the sums do not decrease
    return idx;
}

} // namespace dxmc_gb300::dev
