// Photon-transport kernels for sm_103a.
//
// One persistent launch per job: every lane owns one photon history at a
// time and, inside a warp-synchronous loop, takes a burst of Woodcock steps per
// iteration.  Lanes whose history ended take a photon from a pool that the
// whole warp fills together, so warps stay full until the job runs dry.
// Physics follows DXMClib's
// Transport<T> (include/dxmc/transport.hpp) function by function; each
// device function names the reference lines it restates.
#include "transport.cuh"

#include <algorithm>
#include <mutex>
#include <unordered_map>

namespace dxmc_gb300::dev {

namespace {

    constexpr unsigned FULL_MASK = 0xffffffffu;
    constexpr uint32_t MAX_STEPS_PER_HISTORY = 1u << 20; // guard against unbounded histories

    template <class Real>
    struct PhotonT {
        Real px, py, pz;
        Real dx, dy, dz;
        Real energy;
        Real weight;
    };

    // ---- scoring (transport.hpp:208-214, 598-609) ------------------------------
    // Atomic additions to the tally with an L2 evict-first policy: the tally is
    // read-modify-written at random voxels and would otherwise push the voxel and
    // majorant grids (gathered on every flight) out of L2.
    __device__ __forceinline__ void score_record(TallyRecord* r, double e, double e2, uint32_t n)
    {
#ifdef DXMC_TALLY_NO_HINT
        atomicAdd(&r->energy, e);
        atomicAdd(&r->energy2, e2);
        atomicAdd(&r->events, n);
#else
        asm volatile("{\n\t.reg .b64 pol;\n\tcreatepolicy.fractional.L2::evict_first.b64 pol, 1.0;\n\t"
                     "red.global.add.L2::cache_hint.f64 [%0], %1, pol;\n\t"
                     "red.global.add.L2::cache_hint.f64 [%0+8], %2, pol;\n\t"
                     "red.global.add.L2::cache_hint.u32 [%0+16], %3, pol;\n\t}" ::"l"(r), "d"(e), "d"(e2), "r"(n) : "memory");
#endif
    }

    // The copy of the records that this block adds to.
    __device__ __forceinline__ TallyRecord* tally_records(const TransportParams& p)
    {
        const uint32_t copy = blockIdx.x & (p.tally_copies - 1);
        return copy ? p.more_records + (copy - 1) * p.world.n_voxels : p.records;
    }

    template <bool FAST, class Real>
    __device__ __forceinline__ void score(const TransportParams& p, uint64_t idx, Real e)
    {
        if (FAST || p.records) {
            const double ed = static_cast<double>(e);
            score_record(tally_records(p) + idx, ed, ed * ed, 1u);
            return;
        }
        if constexpr (FAST)
            return;
        if (p.tally_mode == 1) {
            float* t = p.tally_f32 + 2 * idx;
            atomicAdd(t, e);
            atomicAdd(t + 1, e * e);
        } else {
            double* t = p.tally + 2 * idx;
            const double ed = static_cast<double>(e);
            atomicAdd(t, ed);
            atomicAdd(t + 1, ed * ed);
        }
        atomicAdd(p.n_events + idx, 1u);
    }

    // Warp-aggregated scoring: lanes depositing into the same voxel in the same
    // iteration are combined by __match_any_sync and one leader issues the
    // atomics (FP32 partial sums flushed to the FP64 accumulators).
    template <class Real>
    __device__ __forceinline__ void score_aggregated(const TransportParams& p, unsigned active, uint64_t idx, Real e)
    {
        const unsigned peers = __match_any_sync(active, idx);
        const int leader = __ffs(peers) - 1;
        const int lane = threadIdx.x & 31;
        Real sum = Real(0.0), sum2 = Real(0.0);
        unsigned count = 0;
        // each peer group reduces over its members (group sizes are small)
        for (unsigned m = peers; m; m &= m - 1) {
            const int src = __ffs(m) - 1;
            const Real v = __shfl_sync(peers, e, src);
            sum += v;
            sum2 += v * v;
            ++count;
        }
        if (lane == leader) {
            if (p.records) {
                score_record(tally_records(p) + idx, static_cast<double>(sum), static_cast<double>(sum2), count);
            } else {
                double* t = p.tally + 2 * idx;
                atomicAdd(t, static_cast<double>(sum));
                atomicAdd(t + 1, static_cast<double>(sum2));
                atomicAdd(p.n_events + idx, count);
            }
        }
    }

    // Sums and products that the compiler must not fuse: its choice would change with the
    // code around them, and the last bit of a history with it.
    __device__ __forceinline__ float add_rounded(float a, float b) { return __fadd_rn(a, b); }
    __device__ __forceinline__ double add_rounded(double a, double b) { return __dadd_rn(a, b); }
    __device__ __forceinline__ float mul_rounded(float a, float b) { return __fmul_rn(a, b); }
    __device__ __forceinline__ double mul_rounded(double a, double b) { return __dmul_rn(a, b); }

    // The samplers below draw an interaction's outcome (energy imparted, new energy,
    // cosine of the scattering angle); the direction changes in one place for all of
    // them, by an azimuth drawn last (peturb).

    // ---- photoelectric (transport.hpp:216-263) ---------------------------------
    // Returns the energy imparted; `turn`: a characteristic photon of `energy` leaves
    // at angle cosA, otherwise energy is 0.
    template <int MODEL, class Real>
    __device__ __forceinline__ Real photo_sample(const float* L, const LutMeta& m, Real& energy, int material, Rng& rng, Real& cosA, bool& turn)
    {
        const Real E = energy;
        energy = Real(0.0);
        turn = false;
        if constexpr (MODEL < 2) {
            return E;
        } else {
            const float* shells = L + m.off_shells + material * N_SHELLS * SHELL_FLOATS;
            Real cum[N_SHELLS] = {};
            shell_sums<1>(shells, L + m.off_shell_sums + material * SHELL_SUM_FLOATS, E, cum);
            const float* sh = shells + pick_shell(cum, up<Real>(rng.uniform())) * SHELL_FLOATS;
            const Real binding = sh[0];
            if (binding > E || binding < Real(ENERGY_CUTOFF_D))
                return E;
            const Real r1 = up<Real>(rng.uniform());
            if (r1 <= sh[4]) {
                int line = 0;
                Real r3 = up<Real>(rng.uniform()) - sh[5];
                while (r3 > Real(0.0) && line < 2) {
                    ++line;
                    r3 -= sh[5 + line];
                }
                energy = sh[8 + line];
                const Real theta = up<Real>(rng.uniform()) * Real(PI_D);
                cosA = m_cos(theta);
                turn = true;
                return E - energy;
            }
            return E;
        }
    }

    // The whole photoelectric event on a photon, direction included.
    template <int MODEL, class Real>
    __device__ __forceinline__ Real photo_absorption(const float* L, const LutMeta& m, PhotonT<Real>& ph, int material, Rng& rng, bool norm = false)
    {
        Real cosA = Real(1.0);
        bool turn;
        const Real imparted = photo_sample<MODEL>(L, m, ph.energy, material, rng, cosA, turn);
        if (turn) {
            Real sin_phi, cos_phi;
            rng_azimuth(rng, &sin_phi, &cos_phi);
            peturb(ph.dx, ph.dy, ph.dz, cosA, sin_phi, cos_phi, norm);
        }
        return imparted;
    }

    // ---- Rayleigh (transport.hpp:264-298) ---------------------------------------
    template <int MODEL, class Real>
    __device__ __forceinline__ bool rayleigh_sample(const float* G, const LutMeta& m, Real energy, int material, Rng& rng, Real& cosA)
    {
        if constexpr (MODEL == 0) {
            constexpr Real extreme = Real(1.08866210790363); // 4 sqrt(2) / (3 sqrt(3))
            for (int it = 0; it < REJECTION_CAP; ++it) {
                const Real r1 = up<Real>(rng.uniform()) * extreme;
                const Real theta = up<Real>(rng.uniform()) * Real(PI_D);
                Real s, c;
                m_sincos(theta, &s, &c);
                if (!(r1 > (Real(2.0) - s * s) * s)) {
                    cosA = c;
                    return true;
                }
            }
            return false;
        } else {
            // the density of the reference's RITA draw of q^2 <= q_max^2 followed by the
            // (1 + cos^2) / 2 rejection, drawn by inverse CDF: no loop, no divergence
            Real fe;
            const int row = table_row(m, m_log(energy), fe);
            const Real y = table_quantile(G + m.off_ray + (material * m.tab_ne + row) * (m.tab_nu + 1), m.tab_nu, up<Real>(rng.uniform()), fe);
            cosA = Real(1.0) - Real(2.0) * y; // q^2 / q_max^2 = (1 - cos) / 2
            return true;
        }
    }

    // ---- Compton, impulse approximation (transport.hpp:342-483) -----------------
    // The electron shell that takes part, or -1 where the interaction is rejected
    // (no shell can take part, or its binding energy exceeds the photon's).
    template <class Real>
    __device__ __forceinline__ int compton_shell(const float* L, const LutMeta& m, Real energy, int material, Rng& rng)
    {
        const float* shells = L + m.off_shells + material * N_SHELLS * SHELL_FLOATS;
        Real cum[N_SHELLS] = {};
        shell_sums<0>(shells, L + m.off_shell_sums + material * SHELL_SUM_FLOATS, energy, cum);
        const int shell = pick_shell(cum, up<Real>(rng.uniform()));
        if (!(cum[N_SHELLS - 1] > Real(0.0)))
            return -1;
        const Real U = shells[shell * SHELL_FLOATS] / Real(ELECTRON_REST_MASS_D);
        return U > energy / Real(ELECTRON_REST_MASS_D) ? -1 : shell; // the rejection corrects the cross section
    }

    // The rejection draws of a Compton event with the impulse approximation, in two steps
    // so that a warp can repeat the first, cheap one for its rejected lanes and run the
    // second with most of its lanes (both draw in the order of the reference's loop).
    // Which products are fused into sums is written out where it is the compiler's choice,
    // so that every kernel takes the same decisions.
    //
    // First: the energy fraction e from the Klein-Nishina cross section, and t = 1 - cos.
    template <class Real>
    __device__ __forceinline__ bool compton_ia_energy(Real energy, Rng& rng, Real& e, Real& t)
    {
        const Real k = energy / Real(ELECTRON_REST_MASS_D);
        const Real emin = Real(1.0) / (Real(1.0) + Real(2.0) * k);
        const Real gmax_inv = Real(1.0) / (Real(1.0) / emin + emin);
        const Real r1 = up<Real>(rng.uniform());
        // e = r1 + (1 - r1) emin, with 1 - e = (1 - r1)(1 - emin) formed directly so
        // that t stays positive when e rounds to 1 in single precision
        const Real one_minus_e = (Real(1.0) - r1) * (Real(1.0) - emin);
        e = Real(1.0) - one_minus_e;
        t = one_minus_e / (k * e);
        const Real sin2 = mul_rounded(t, (Real(2.0) - t));
        const Real g = add_rounded(Real(1.0) / e + e, -sin2) * gmax_inv;
        const Real r2 = up<Real>(rng.uniform());
        return !(r2 > g);
    }

    // Second: the electron's momentum in shell `sh`; where it accepts, e with the Doppler
    // shift and the angle.
    template <class Real>
    __device__ __forceinline__ bool compton_ia_shift(const float* sh, Real energy, Rng& rng, Real t, Real& e, Real& cosA)
    {
        const Real U = sh[0] / Real(ELECTRON_REST_MASS_D);
        const Real pU = m_sqrt(m_fma(U, U, Real(2.0) * U));
        const Real J0 = sh[2];
        const Real k = energy / Real(ELECTRON_REST_MASS_D);
        constexpr Real sp2 = Real(2.50662827463100); // 1 / (1/sqrt(pi) / sqrt(2)) = sqrt(2 pi)
        constexpr Real a1 = Real(0.34802), a2 = -Real(0.0958798), a3 = Real(0.7478556);
        const Real sqrte = Real(1.64872127070013);
        const Real sin2 = t * (Real(2.0) - t);
        cosA = Real(1.0) - t;
        const Real kU = k * (k - U);
        const Real pi = m_fma(kU, t, -U) / m_sqrt(m_max(m_fma(U, U, Real(2.0) * mul_rounded(kU, t)), Real(1e-30)));
        const Real kc = k * e;
        const Real qc = m_sqrt(m_max(m_fma(Real(-2.0) * k * kc, cosA, m_fma(k, k, mul_rounded(kc, kc))), Real(1e-30)));
        const Real alpha = qc * (Real(1.0) + kc * (kc - k * cosA) / (qc * qc)) / k;
        const Real b_part = Real(1.0) + Real(2.0) * J0 * m_abs(pi);
        const Real b = (b_part * b_part + Real(1.0)) * Real(0.5);
        const Real expb = m_exp(-b);
        Real S;
        if (pi <= -pU) {
            S = (Real(1.0) - alpha * pU) * expb * Real(0.5);
        } else if (pi < pU) {
            const Real part1 = alpha * sp2 / (Real(4.0) * J0);
            const Real tp = Real(1.0) / (Real(1.0) + Real(0.332673) * (Real(1.0) + Real(2.0) * J0 * m_abs(pU)));
            const Real tpi = Real(1.0) / (Real(1.0) + Real(0.332673) * (Real(1.0) + Real(2.0) * J0 * m_abs(pi)));
            const Real part2p = m_fma(-(expb * tp), m_fma(a3 * tp, tp, m_fma(a2, tp, a1)), sqrte);
            const Real part2pi = m_fma(-(expb * tpi), m_fma(a3 * tpi, tpi, m_fma(a2, tpi, a1)), sqrte);
            const Real D = add_rounded(part2p, -part2pi);
            const Real X5 = mul_rounded(m_fma(-alpha, pi, Real(1.0)), expb) * Real(0.5);
            if (pi <= Real(0.0))
                S = add_rounded(X5, -mul_rounded(part1, D));
            else
                S = m_fma(-part1, D, add_rounded(Real(1.0), -X5));
        } else {
            S = Real(1.0) - (Real(1.0) - alpha * pU) * expb * Real(0.5);
        }
        const Real r3 = up<Real>(rng.uniform());
        if (r3 > S)
            return false;
        Real Fmax;
        if (pi <= -pU)
            Fmax = Real(1.0) - alpha * pU;
        else if (pi >= pU)
            Fmax = Real(1.0) + alpha * pU;
        else
            Fmax = Real(1.0) + alpha * pi;
        const Real r4 = up<Real>(rng.uniform_open()); // log(rbar2) below needs rbar2 > 0
        const Real rbar2 = Real(2.0) * r4 * expb;
        Real pz;
        if (rbar2 < Real(1.0)) {
            const Real part = m_sqrt(Real(1.0) - Real(2.0) * m_log(rbar2));
            pz = (Real(1.0) - part) / (Real(2.0) * J0) / Real(ELECTRON_REST_MASS_D);
        } else {
            const Real part = m_sqrt(Real(1.0) - Real(2.0) * m_log(Real(2.0) - rbar2));
            pz = (part - Real(1.0)) / (Real(2.0) * J0) / Real(ELECTRON_REST_MASS_D);
        }
        Real Fpz;
        if (pz <= -pU)
            Fpz = Real(1.0) - alpha * pU;
        else if (pz >= pU)
            Fpz = Real(1.0) + alpha * pU;
        else
            Fpz = Real(1.0) + alpha * pz;
        const Real r5 = up<Real>(rng.uniform());
        if (r5 > Fpz / Fmax)
            return false;
        const Real part = m_sqrt(m_max(Real(1.0) - Real(2.0) * e * cosA + e * e * (Real(1.0) - pz * pz * sin2), Real(0.0)));
        const Real kbar = kc / (Real(1.0) - pz * pz * e * e) * (Real(1.0) - pz * pz * e * cosA + pz * part);
        e = kbar / k;
        return true;
    }

    template <class Real>
    __device__ __forceinline__ bool compton_ia(const float* sh, Real energy, Rng& rng, Real& e, Real& cosA)
    {
        for (int it = 0; it < REJECTION_CAP; ++it) {
            Real t;
            if (compton_ia_energy(energy, rng, e, t) && compton_ia_shift(sh, energy, rng, t, e, cosA))
                return true;
        }
        return false;
    }

    // ---- Compton, Klein-Nishina with optional scatter factor (transport.hpp:300-340)
    // Energy fraction and angle from the quantile x = (e - e_min) / (1 - e_min).
    template <class Real>
    __device__ __forceinline__ void compton_from_fraction(Real E, Real x, Real& e, Real& cosA)
    {
        const Real k = E / Real(ELECTRON_REST_MASS_D);
        const Real emin = Real(1.0) / (Real(1.0) + Real(2.0) * k);
        const Real one_minus_e = (Real(1.0) - x) * (Real(1.0) - emin);
        e = Real(1.0) - one_minus_e;
        cosA = m_max(Real(1.0) - one_minus_e / (k * e), -Real(1.0));
    }

    // Returns false where the sampling loop hit its cap; `turn` false: the interaction
    // was rejected (nothing changes, zero energy imparted).
    template <int MODEL, class Real>
    __device__ __forceinline__ bool compton_sample(const float* L, const float* G, const LutMeta& m, Real& energy, int material, Rng& rng, Real& cosA,
        Real& imparted, bool& turn)
    {
        const Real E = energy;
        imparted = Real(0.0);
        turn = true;
        Real e;
        if constexpr (MODEL == 2) {
            const int shell = compton_shell(L, m, E, material, rng);
            if (shell < 0) {
                turn = false;
                return true;
            }
            e = Real(1.0);
            if (!compton_ia(L + m.off_shells + (material * N_SHELLS + shell) * SHELL_FLOATS, E, rng, e, cosA))
                return false;
        } else {
            // the density of the reference's Klein-Nishina rejection (times the scatter
            // factor S(q) for LIVERMORE), drawn by inverse CDF: no loop, no divergence
            Real fe;
            const int row = table_row(m, m_log(E), fe);
            const float* tab = MODEL == 1 ? G + m.off_csf + (material * m.tab_ne + row) * (m.tab_nu + 1)
                                          : G + m.off_ckn + row * (m.tab_nu + 1);
            const Real x = table_quantile(tab, m.tab_nu, up<Real>(rng.uniform()), fe);
            compton_from_fraction(E, x, e, cosA);
        }
        energy = E * e;
        imparted = E - energy;
        return true;
    }

    // ---- photon generation: Exposure::sampleParticle (exposure.hpp:280-304) -----
    template <class Real>
    __device__ __forceinline__ void sample_particle(const SourceParams& s, const DevExposure& ex, Rng& rng, PhotonT<Real>& ph)
    {
        const Real theta = up<Real>(ex.coll[0]) + up<Real>(rng.uniform()) * up<Real>(ex.coll[1] - ex.coll[0]);
        const Real phi = up<Real>(ex.coll[2]) + up<Real>(rng.uniform()) * up<Real>(ex.coll[3] - ex.coll[2]);
        ph.px = up<Real>(ex.pos[0]);
        ph.py = up<Real>(ex.pos[1]);
        ph.pz = up<Real>(ex.pos[2]);
        ph.dx = up<Real>(ex.beam[0]);
        ph.dy = up<Real>(ex.beam[1]);
        ph.dz = up<Real>(ex.beam[2]);
        ph.weight = up<Real>(ex.weight);
        rotate(ph.dx, ph.dy, ph.dz, up<Real>(ex.cosy[0]), up<Real>(ex.cosy[1]), up<Real>(ex.cosy[2]), theta);
        rotate(ph.dx, ph.dy, ph.dz, up<Real>(ex.cosx[0]), up<Real>(ex.cosx[1]), up<Real>(ex.cosx[2]), phi);
        if (s.spec_n > 0) {
            // SpecterDistribution::sampleValue (dxmcrandom.hpp:322-326)
            const Real r = up<Real>(rng.uniform());
            const uint32_t k = rng.below(static_cast<uint32_t>(s.spec_n));
            const uint32_t idx = r < up<Real>(__ldg(s.spec_prob + k)) ? k : __ldg(s.spec_alias + k);
            if (idx + 1 < static_cast<uint32_t>(s.spec_n)) {
                const Real e0 = up<Real>(__ldg(s.spec_energy + idx)), e1 = up<Real>(__ldg(s.spec_energy + idx + 1));
                ph.energy = e0 + up<Real>(rng.uniform()) * (e1 - e0);
            } else {
                ph.energy = up<Real>(__ldg(s.spec_energy + idx));
            }
        } else {
            ph.energy = up<Real>(ex.mono_energy);
        }
        if (s.bowtie_angle) {
            // BowTieFilter::sampleIntensityWeight (beamfilters.hpp:150-190)
            const Real angle = m_abs(theta);
            int first = 0, last = s.bowtie_n - 1;
            int it = first + (last - first) / 2;
            while (it != first) {
                if (angle < __ldg(s.bowtie_angle + it)) {
                    last = it;
                    it = first;
                } else {
                    first = it;
                }
                it += (last - first) / 2;
            }
            Real w;
            if (angle < __ldg(s.bowtie_angle + first))
                w = __ldg(s.bowtie_weight);
            else if (angle > __ldg(s.bowtie_angle + last))
                w = __ldg(s.bowtie_weight + s.bowtie_n - 1);
            else {
                const Real x0 = __ldg(s.bowtie_angle + first), x1 = __ldg(s.bowtie_angle + last);
                const Real y0 = __ldg(s.bowtie_weight + first), y1 = __ldg(s.bowtie_weight + last);
                w = y0 + (angle - x0) * (y1 - y0) / (x1 - x0);
            }
            ph.weight *= w;
        }
        if (s.heel_weights) {
            // HeelFilter::sampleIntensityWeight (beamfilters.hpp:514-538)
            const Real energy = ph.energy;
            int e_index = static_cast<int>((energy - up<Real>(s.heel_e_start) + Real(0.5) * up<Real>(s.heel_e_step)) / up<Real>(s.heel_e_step));
            if (e_index >= s.heel_e_size || e_index < 0)
                e_index = e_index < 0 ? 0 : s.heel_e_size - 1;
            if (energy < up<Real>(s.heel_e_start))
                e_index = 0;
            int a_index = static_cast<int>((phi - up<Real>(s.heel_a_start)) / up<Real>(s.heel_a_step));
            if (a_index >= s.heel_a_size || a_index < 0)
                a_index = a_index < 0 ? 0 : s.heel_a_size - 1;
            if (phi < up<Real>(s.heel_a_start))
                a_index = 0;
            const int w_index = e_index * s.heel_a_size + a_index;
            Real w;
            if (a_index < s.heel_a_size - 1) {
                const Real a0 = up<Real>(s.heel_a_start + s.heel_a_step * a_index);
                const Real a1 = up<Real>(s.heel_a_start + s.heel_a_step * (a_index + 1));
                const Real w0 = up<Real>(__ldg(s.heel_weights + w_index)), w1 = up<Real>(__ldg(s.heel_weights + w_index + 1));
                w = w0 + (w1 - w0) * (phi - a0) / (a1 - a0);
            } else {
                w = up<Real>(__ldg(s.heel_weights + w_index));
            }
            ph.weight *= w;
        }
    }

    template <class Real>
    __device__ __forceinline__ bool inside(const WorldParams& w, Real x, Real y, Real z)
    {
        return (x > up<Real>(w.lo[0]) && x < up<Real>(w.hi[0])) && (y > up<Real>(w.lo[1]) && y < up<Real>(w.hi[1])) && (z > up<Real>(w.lo[2]) && z < up<Real>(w.hi[2]));
    }

    // transportParticleToWorld (transport.hpp:702-728)
    template <class Real>
    __device__ __forceinline__ bool transport_to_world(const WorldParams& w, PhotonT<Real>& ph)
    {
        if (inside(w, ph.px, ph.py, ph.pz))
            return true;
        Real amin = -Real(3.402823466e38), amax = Real(3.402823466e38);
        const Real pos[3] = { ph.px, ph.py, ph.pz };
        const Real dir[3] = { ph.dx, ph.dy, ph.dz };
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            if (m_abs(dir[i]) > Real(N_ERROR_D)) {
                const Real inv = Real(1.0) / dir[i];
                const Real a0 = (up<Real>(w.lo[i]) - pos[i]) * inv;
                const Real an = (up<Real>(w.hi[i]) - pos[i]) * inv;
                amin = m_max(amin, m_min(a0, an));
                amax = m_min(amax, m_max(a0, an));
            }
        }
        if (amin < amax && amin > Real(0.0)) {
            ph.px += amin * ph.dx;
            ph.py += amin * ph.dy;
            ph.pz += amin * ph.dz;
            return true;
        }
        return false;
    }

    __device__ __forceinline__ uint32_t find_exposure(const SourceParams& s, uint64_t h)
    {
        // last exposure whose offset <= h
        uint32_t lo = 0, hi = s.n_exposures;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (__ldg(s.history_offsets + mid) <= h)
                lo = mid;
            else
                hi = mid;
        }
        return lo;
    }

    __device__ __forceinline__ void load_exposure(const DevExposure* ptr, DevExposure& ex)
    {
        const float4* src = reinterpret_cast<const float4*>(ptr);
        float4* dst = reinterpret_cast<float4*>(&ex);
#pragma unroll
        for (int i = 0; i < 5; ++i)
            dst[i] = __ldg(src + i);
    }

    // A voxel as read from the grid: its palette index (compact layout) or its
    // 8-byte record; decode_voxel turns it into density, material and the
    // measurement flag.  Compact worlds hold fewer than 2^32 voxels (world upload),
    // so their voxel index is 32 bits.
    template <bool PALETTE>
    struct VoxelRaw {
        using Index = uint64_t;
        uint2 v;
    };
    template <>
    struct VoxelRaw<true> {
        using Index = uint32_t;
        uint32_t index;
    };

    template <bool PALETTE>
    __device__ __forceinline__ typename VoxelRaw<PALETTE>::Index voxel_index(const WorldParams& w, uint32_t ix, uint32_t iy, uint32_t iz)
    {
        using Index = typename VoxelRaw<PALETTE>::Index;
        if constexpr (PALETTE)
            return iz * static_cast<uint32_t>(w.nxy) + (iy * w.dims[0] + ix);
        else
            return static_cast<Index>(iz) * w.nxy + static_cast<Index>(iy) * w.dims[0] + ix;
    }

    template <bool PALETTE>
    __device__ __forceinline__ VoxelRaw<PALETTE> load_voxel(const WorldParams& w, typename VoxelRaw<PALETTE>::Index vidx)
    {
        if constexpr (PALETTE)
            return VoxelRaw<true> { __ldg(w.palette_index + vidx) };
        else
            return VoxelRaw<false> { __ldg(reinterpret_cast<const uint2*>(w.voxels) + vidx) };
    }

    template <bool PALETTE, class Real>
    __device__ __forceinline__ void decode_voxel(const VoxelRaw<PALETTE>& raw, const PaletteEntry* pal, Real& density, int& mat, bool& measured)
    {
        if constexpr (PALETTE) {
            const PaletteEntry e = pal[raw.index];
            density = up<Real>(e.density);
            mat = static_cast<int>(e.code & 0xffu);
            measured = (e.code >> 8) != 0u;
        } else {
            density = up<Real>(__uint_as_float(raw.v.x));
            mat = static_cast<int>(raw.v.y & 0xffu);
            measured = ((raw.v.y >> 8) & 0xffu) != 0u;
        }
    }

#ifndef DXMC_MIN_BLOCKS_PER_SM
#define DXMC_MIN_BLOCKS_PER_SM 4 // resident blocks per SM the register budget must allow (64 or 56 registers, see transport_block)
#endif

    // Flights per iteration of the loop.  A lane that stops waits for the end of the burst,
    // and a flight costs the warp the same whatever its lanes: where most flights end in an
    // event or outside the grid (radiography, CTDI: 0.9 stops per flight) two are best, in
    // a body with air and lung (CT: 0.4) four.  Unless the job sets it, a warp takes
    // START_BURST and then goes by the stops per flight it has seen.  A vote of the warp
    // after each flight, to stop when few lanes were left, cost more than it saved.
    // CT 512 x 512 x 100 of 2e7 histories with bursts of 2 / 3 / 4 / 5: 2.49 / 2.42 / 2.41 /
    // 2.45 ms (2.52 voting); DX 160^3 of 5e6: 0.570 / 0.588 / 0.600 / 0.61 ms (0.587).
    constexpr int START_BURST = 3; // FP64: SHORT_BURST, each of its flights costs more
    constexpr int SHORT_BURST = 2, LONG_BURST = 4;
    constexpr uint32_t LONG_BURST_STOPS = 55; // per hundred flights, at most

    // Histories between two additions of a warp's counters to the job's (its progress while
    // it runs): the counters share a line with the queue's head.
    constexpr uint32_t PUBLISH_HISTORIES = 4096;

    // What belongs to a warp rather than to a lane, in shared memory: in registers every
    // lane would hold a copy through the whole loop (a dozen of its 64).
    struct WarpState {
        uint64_t next, end;                      // ids [next, end) to sample
        int pooled;                              // photons in the pool
        uint32_t steps, deposits, histories;     // since they were last added to the job's counters
        unsigned int overflows, forced_deposits; // rare events, by shared atomics
        int burst;                               // flights per iteration
        uint64_t carried[3];                     // steps, histories and deposits beyond 32 bits
    };

    // A warp's counters are 32 bits wide, a job's 64: lane 0 empties them, between units of work,
    // once one is beyond CARRY, while the steps of a unit and of the photons in flight still
    // fit (and the burst's rule, in 32 bits as well).
    constexpr uint32_t CARRY = 1u << 24;
    static_assert(CARRY + (256 + 2 * 32) * (MAX_STEPS_PER_HISTORY + 64ull) <= 0xffffffffull, "no counter of a warp wraps");
    __device__ __forceinline__ void carry_counters(WarpState& ws)
    {
        if ((ws.histories | ws.steps) >= CARRY) {
            ws.carried[0] += ws.steps;
            ws.carried[1] += ws.histories;
            ws.carried[2] += atomicExch(&ws.deposits, 0u); // the lanes add to it
            ws.carried[2] += atomicExch(&ws.forced_deposits, 0u);
            ws.steps = ws.histories = 0;
        }
    }

    // Adds the warp's counters to the job's and clears them.  Called by all 32 lanes.
    __device__ __forceinline__ void add_counters(WarpState& ws, JobCounters* c)
    {
        __syncwarp();
        if ((threadIdx.x & 31) == 0) {
            const uint64_t steps = ws.carried[0] + ws.steps, histories = ws.carried[1] + ws.histories;
            const uint64_t deposits = ws.carried[2] + ws.deposits + ws.forced_deposits;
            if (steps)
                atomicAdd(&c->steps, static_cast<unsigned long long>(steps));
            if (deposits)
                atomicAdd(&c->deposits, static_cast<unsigned long long>(deposits));
            if (ws.overflows)
                atomicAdd(&c->overflows, static_cast<unsigned long long>(ws.overflows));
            if (histories)
                atomicAdd(&c->histories_done, static_cast<unsigned long long>(histories));
            ws.carried[0] = ws.carried[1] = ws.carried[2] = 0;
            ws.steps = ws.deposits = ws.histories = 0;
            ws.overflows = ws.forced_deposits = 0;
        }
        __syncwarp();
    }

    // What a lane does: it flies, it waits for a stage of the loop, or it waits for the
    // event of a real collision in the material |state| - 1 (negative: at a forced-scoring
    // voxel).  The event's type is drawn in the interaction pass, where more lanes share
    // the work than in the flight loop.
    constexpr int FLYING = 0;
    constexpr int IDLE = 0x200;  // no photon
    constexpr int SETUP = 0x201; // new photon or energy: majorant, attenuation and cell to look up
    constexpr int REACH = 0x202; // the next flight leaves the ball of its cell outside the body box

    // A Compton event of the impulse approximation whose draws were rejected so far (the
    // negative of it: at a forced-scoring voxel), TRYING | shell | draws << TRY_SHIFT with
    // `shell` counted over all materials.
    constexpr int TRYING = 0x1000;
    constexpr int TRY_SHIFT = 13;
    static_assert(256 * N_SHELLS <= TRYING && (static_cast<int64_t>(REJECTION_CAP) << TRY_SHIFT) < 0x7fffffff, "the state holds shell and draws");
    // A pass repeats the energy draws while MIN_TRYING lanes are rejected and whole rounds
    // of draws while MIN_ROUND lanes are; the others join the next pass.  One draw in five
    // is accepted.  DX 127^3, 4e6 histories, rounds down to 33 / 20 / 16 / 12 / 8 lanes:
    // 1.44 / 1.40 / 1.31 / 1.26 / 1.27 ms (1.18 ms with the LUT's partial sums of the shells).
    constexpr int MIN_TRYING = 2;
    constexpr int MIN_ROUND = 12;

    __device__ __forceinline__ bool waits_for_event(int state) { return state != FLYING && (state < IDLE || state >= TRYING); }

    // State of one lane: its photon, random stream and cached lookups.
    template <class Real, class Index>
    struct LaneT {
        PhotonT<Real> ph;
        Rng rng;
        int state;
        Real stepK; // Woodcock step = -log2(u) * stepK (mm): 10 * ln 2 / majorant
        uint32_t hist_steps;
        Index vidx;
        bool armed;      // energy x weight is below the Russian-roulette threshold
        Real cinv, cR;  // local majorant: 1 / scale and the flight length it holds for (MajorantGrid)
        int band;        // energy band of the local-majorant grid
        // without the attenuation table: the last material met at this energy
        Real logE;
        int seg;
        int cached_mat;
        Real probInv;   // attenuation of the material / majorant (event probability per unit density)
        Real p0, p01;   // FP64: photoelectric and photoelectric + Compton shares of the attenuation
        Real forced_wc; // weight correction waiting for a forced-voxel interaction pass

        __device__ void start_photon()
        {
            state = SETUP;
            cached_mat = -1;
            hist_steps = 0;
            forced_wc = Real(0.0);
            cinv = Real(1.0); // the first flight from the grid boundary uses the global majorant
            cR = INFINITY;
            arm();
        }
        // energy and weight change only at interactions and roulette: the roulette
        // test of a virtual step reads this flag
        __device__ void arm() { armed = ph.energy * ph.weight < Real(ROULETTE_THRESHOLD_D); }
    };

    // Local majorant of the photon's cell for its energy band, after the energy
    // changed (a new photon, or an interaction): the flight drawn next must be
    // bounded for the new energy.  A new photon sits on the grid boundary, so the
    // coordinates are clamped onto the grid.
    template <class Real, class Index>
    __device__ __forceinline__ void fetch_cell(LaneT<Real, Index>& s, const TransportParams& p, Real logE)
    {
        const MajorantGrid& g = p.majorant;
        const WorldParams& w = p.world;
        // the band intervals of the bounds are widened by 0.1 % on the host, which
        // covers the rounding here
        s.band = min(max(m_floor_int((logE - up<Real>(g.band_log0)) * up<Real>(g.band_inv_dlog)), 0), g.bands - 1);
        const Real fx = m_min(m_max(m_fma(s.ph.px, up<Real>(w.inv_spacing[0]), -up<Real>(w.lo_inv[0])), Real(0.0)), up<Real>(w.dims_f[0]) - Real(1.0));
        const Real fy = m_min(m_max(m_fma(s.ph.py, up<Real>(w.inv_spacing[1]), -up<Real>(w.lo_inv[1])), Real(0.0)), up<Real>(w.dims_f[1]) - Real(1.0));
        const Real fz = m_min(m_max(m_fma(s.ph.pz, up<Real>(w.inv_spacing[2]), -up<Real>(w.lo_inv[2])), Real(0.0)), up<Real>(w.dims_f[2]) - Real(1.0));
        const uint32_t ix = static_cast<uint32_t>(fx), iy = static_cast<uint32_t>(fy), iz = static_cast<uint32_t>(fz);
        const uint32_t c = (iz >> g.shift[2]) * g.nxy + (iy >> g.shift[1]) * g.nx + (ix >> g.shift[0]);
        const float2 cell = __ldg(g.cells + (c * g.bands + s.band));
        s.cinv = up<Real>(cell.x);
        s.cR = up<Real>(cell.y);
    }

    // Safe flight length in a cell outside the box of the denser cells (the cell
    // holds -R): the ball of radius R, or the ray up to where it enters the box
    // (slab test in flight-parameter units, as the position update), whichever
    // reaches further.  A ray that misses the box may fly to the grid boundary.
    template <class Real>
    __device__ __forceinline__ Real reach_to_box(const PhotonT<Real>& ph, const MajorantGrid& g, Real R)
    {
        const Real p[3] = { ph.px, ph.py, ph.pz };
        const Real d[3] = { ph.dx, ph.dy, ph.dz };
        Real tmin = Real(0.0), tmax = INFINITY;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const Real inv = Real(1.0) / d[a];
            const Real t0 = (up<Real>(g.box_lo[a]) - p[a]) * inv;
            const Real t1 = (up<Real>(g.box_hi[a]) - p[a]) * inv;
            tmin = m_max(tmin, m_min(t0, t1));
            tmax = m_min(tmax, m_max(t0, t1));
        }
        return m_max(R, tmin <= tmax ? tmin : INFINITY);
    }

    // Loads photon + stream state from the pre-generated queue.
    template <class Real>
    __device__ __forceinline__ void load_queued(PhotonT<Real>& ph, Rng& rng, const PhotonQueue& q, uint64_t i)
    {
        const float4 pe = __ldg(q.pos_energy + i);
        const float4 dw = __ldg(q.dir_weight + i);
        const uint4 rs = __ldg(q.rng + i);
        ph = PhotonT<Real> { pe.x, pe.y, pe.z, dw.x, dw.y, dw.z, pe.w, dw.w };
        rng.s0 = rs.x;
        rng.s1 = rs.y;
        rng.s2 = rs.z;
        rng.s3 = rs.w;
    }

    // Samples history h of the job (Exposure::sampleParticle); false: it misses the
    // grid (transportParticleToWorld).
    template <class Real>
    __device__ __forceinline__ bool sample_history(PhotonT<Real>& ph, Rng& rng, const TransportParams& p, uint64_t h)
    {
        rng.init_keyed(p.stream_key, h);
        uint32_t ei;
        if (p.uniform_hpe && p.total_histories <= 0xffffffffull)
            ei = udiv_apply(static_cast<uint32_t>(h), p.hpe_magic, p.hpe_shifts);
        else
            ei = p.uniform_hpe ? static_cast<uint32_t>(h / p.uniform_hpe) : find_exposure(p.source, h);
        DevExposure ex;
        load_exposure(p.source.exposures + ei, ex);
        sample_particle(p.source, ex, rng, ph);
        return transport_to_world(p.world, ph);
    }

    template <class Real, class Index>
    __device__ __forceinline__ void take_history(LaneT<Real, Index>& s, const TransportParams& p, uint64_t h)
    {
        const bool inside = sample_history(s.ph, s.rng, p, h);
        s.start_photon();
        if (!inside)
            s.state = IDLE;
    }

    // The lanes of a warp for next_ids.
    struct DeviceWarp {
        __device__ __forceinline__ bool leader() const { return (threadIdx.x & 31) == 0; }
        __device__ __forceinline__ void sync() const { __syncwarp(); }
        __device__ __forceinline__ uint64_t broadcast(uint64_t v) const { return __shfl_sync(FULL_MASK, v, 0); }
        __device__ __forceinline__ uint64_t fetch_add(unsigned long long* head) const { return atomicAdd(head, 1ull); }
        __device__ __forceinline__ void stop(unsigned long long* head) const { atomicOr(head, static_cast<unsigned long long>(QUEUE_STOPPED)); }
    };

    // Photons sampled ahead for one warp (shared memory, one row per field).  All 32
    // lanes sample together, whatever their own photons do; idle lanes then take photons
    // from here.  Sampling in place, 13 lanes at a time, took 20 % of the instructions
    // of the CT workload.
    template <class Real>
    struct PhotonPool {
        struct alignas(4 * sizeof(Real)) Quad {
            Real v[4];
        };
        Quad position[32]; // and energy
        Quad direction[32]; // and weight
        uint4 rng[32];

        __device__ __forceinline__ void put(int i, const PhotonT<Real>& ph, const Rng& r)
        {
            position[i] = Quad { { ph.px, ph.py, ph.pz, ph.energy } };
            direction[i] = Quad { { ph.dx, ph.dy, ph.dz, ph.weight } };
            rng[i] = make_uint4(r.s0, r.s1, r.s2, r.s3);
        }
        __device__ __forceinline__ void get(int i, PhotonT<Real>& ph, Rng& r) const
        {
            const Quad a = position[i], b = direction[i];
            const uint4 q = rng[i];
            ph = PhotonT<Real> { a.v[0], a.v[1], a.v[2], b.v[0], b.v[1], b.v[2], a.v[3], b.v[3] };
            r.s0 = q.x;
            r.s1 = q.y;
            r.s2 = q.z;
            r.s3 = q.w;
        }
    };

    // In double precision the three exponentials of the shares cost more than two
    // registers: the shares of the event types stay with the cached material.
    template <class Real, bool FAST>
    constexpr bool keeps_shares = !FAST && sizeof(Real) == 8;

    // attenuation (1 / cm) x stepK (mm) -> event probability
    template <class Real>
    constexpr Real per_step = Real(1.0) / (Real(10.0) * Real(0.693147180559945));

    // Photoelectric share, and photoelectric + Compton share, of a material's attenuation.
    template <class Real>
    __device__ __forceinline__ void type_shares(const float* L, const LutMeta& m, int mat, Real energy, Real& p0, Real& p01)
    {
        const Real logE = m_log10(energy);
        Real a0, a1, a2;
        lut_attenuation(L, m, mat, logE, lut_segment(L, m, logE), a0, a1, a2);
        const Real inv = Real(1.0) / (a0 + a1 + a2);
        p0 = a0 * inv;
        p01 = (a0 + a1) * inv;
    }

    // Russian roulette (transport.hpp:684-694) after an interaction or a forced step.
    template <class Real, class Index>
    __device__ __forceinline__ void roulette(LaneT<Real, Index>& s)
    {
        if (s.ph.energy * s.ph.weight < Real(ROULETTE_THRESHOLD_D)) {
            if (up<Real>(s.rng.uniform()) < Real(ROULETTE_PROBABILITY_D))
                s.state = IDLE;
            else
                s.ph.weight *= Real(1.0) / (Real(1.0) - Real(ROULETTE_PROBABILITY_D));
        }
        s.arm();
    }

    // The collision test at the end of a flight drawn with the majorant scale 1 / cinv:
    // a real event (the lane waits for the interaction pass), a virtual collision with
    // Russian roulette, or the forced scoring of a measurement voxel.
    template <int MODEL, bool PALETTE, bool FORCED, bool FAST, class Real, class Index>
    __device__ __forceinline__ void collide(LaneT<Real, Index>& s, WarpState& ws, const TransportParams& p, const float* L, const PaletteEntry* pal,
        const float* table, const VoxelRaw<PALETTE>& raw, Real cinv)
    {
        const LutMeta& m = p.lut_meta;
        constexpr bool SHARES = keeps_shares<Real, FAST>;
        Real density;
        int mat;
        bool measured;
        decode_voxel<PALETTE>(raw, pal, density, mat, measured);
        Real probInv;
        if constexpr (FAST) {
            probInv = table[mat * ATT_TABLE_LANES];
        } else {
            if (mat != s.cached_mat) {
                Real a0, a1, a2;
                lut_attenuation(L, m, mat, s.logE, s.seg, a0, a1, a2);
                const Real total = a0 + a1 + a2;
                s.probInv = total * s.stepK * per_step<Real>;
                s.cached_mat = mat;
                if constexpr (SHARES) {
                    const Real inv = Real(1.0) / total;
                    s.p0 = a0 * inv;
                    s.p01 = (a0 + a1) * inv;
                }
            }
            probInv = s.probInv;
        }
        const Real eventProb = probInv * density * cinv;
        if (!FORCED || !measured) {
            // naive sampling (computeInteractions): the event runs in the interaction pass
            if (up<Real>(s.rng.uniform()) < eventProb) {
                s.state = 1 + mat;
            } else if (s.armed) {
                // virtual collision: Russian roulette (transport.hpp:684-694)
                if (up<Real>(s.rng.uniform()) < Real(ROULETTE_PROBABILITY_D)) {
                    s.state = IDLE;
                } else {
                    s.ph.weight *= Real(1.0) / (Real(1.0) - Real(ROULETTE_PROBABILITY_D));
                    s.arm();
                }
            }
        } else {
            // forced photoelectric scoring (computeInteractionsForced): score the forced
            // photoelectric share now; a real Compton or Rayleigh event goes through the
            // interaction pass and the weight correction (1 - wc) is applied after it
            Real photoProb, unused;
            if constexpr (SHARES)
                photoProb = s.p0;
            else
                type_shares(L, m, mat, s.ph.energy, photoProb, unused);
            const Real wc = eventProb * photoProb;
            PhotonT<Real> forced = s.ph;
            const Real ef = photo_absorption<MODEL>(L, m, forced, mat, s.rng, !FAST && p.normalize_direction);
            const Real forced_deposit = (forced.energy < Real(ENERGY_CUTOFF_D) ? (ef + forced.energy) : ef) * forced.weight * wc;
            if (isfinite(forced_deposit)) {
                score<FAST>(p, s.vidx, forced_deposit);
                atomicAdd(&ws.forced_deposits, 1u);
                if (up<Real>(s.rng.uniform()) < eventProb * (Real(1.0) - photoProb)) {
                    s.forced_wc = wc;
                    s.state = -1 - mat;
                } else {
                    s.ph.weight *= (Real(1.0) - wc);
                    roulette(s);
                }
            } else {
                atomicAdd(&ws.overflows, 1u);
                s.state = IDLE;
            }
        }
    }

    // One iteration of the warp-synchronous loop for every lane of the warp: up to
    // ws.burst Woodcock flights for lanes without a pending event
    // (transport.hpp:650-699), the interaction pass once enough lanes wait
    // (transport.hpp:523-638), Russian roulette and scoring.  Must be called by all 32
    // lanes.
    //
    // FORCED: the world has a measurement map (forced photoelectric scoring); worlds
    // without one run a kernel that does not hold that code.  FAST: the job's options are
    // those of TransportVariant::fast, and `table` (shared memory, one column of lanes per
    // material) holds the event probability per unit density of every material at the
    // lane's energy, filled when the energy changes, with most lanes of the warp in step;
    // otherwise the lane evaluates the material it meets and keeps the last one.  LEAN
    // (the persistent multi-job kernel,
    // which holds more state per lane) reads the voxel after the truncation test.
    template <int MODEL, bool PALETTE, bool FORCED, bool FAST, bool LEAN = false, class Real, class Index>
    __device__ __forceinline__ void advance(LaneT<Real, Index>& s, WarpState& ws, const TransportParams& p, const float* L, const PaletteEntry* pal,
        float* table, bool drain, int interact_t)
    {
        const LutMeta& m = p.lut_meta;
        const WorldParams& w = p.world;
        constexpr bool SHARES = keeps_shares<Real, FAST>;

        // ---- setup -----------------------------------------------------------------------
        if (s.state == SETUP || s.state == REACH) {
            if (s.state == SETUP) {
                const Real logE = m_log10(s.ph.energy);
                const int seg = lut_segment(L, m, logE);
                s.stepK = lut_max_inverse(L, m, logE, seg) * (Real(10.0) * Real(0.693147180559945)); // cm -> mm, log2 -> ln
                // the cell is read before the attenuations, whose arithmetic hides its latency
                if (FAST || p.majorant.cells)
                    fetch_cell(s, p, logE);
                if constexpr (FAST) {
                    for (int mat = 0; mat < m.n_materials; ++mat) {
                        Real a0, a1, a2;
                        lut_attenuation(L, m, mat, logE, seg, a0, a1, a2);
                        table[mat * ATT_TABLE_LANES] = (a0 + a1 + a2) * s.stepK * per_step<Real>;
                    }
                } else {
                    s.logE = logE;
                    s.seg = seg;
                    s.cached_mat = -1;
                }
            }
            // the slab test of the body box runs here, once per iteration for every lane
            // that needs it: in the flight loop 6 of 18 lanes took it in nearly every
            // flight, 22 % of the instructions of the CT workload
            if (s.cR < Real(0.0))
                s.cR = reach_to_box(s.ph, p.majorant, -s.cR);
            s.state = FLYING;
        }
        if (s.state == FLYING && s.hist_steps > MAX_STEPS_PER_HISTORY) {
            // bounded work per history (checked per burst: at most burst - 1 steps over)
            atomicAdd(&ws.overflows, 1u);
            s.state = IDLE;
        }

        // ---- flights ---------------------------------------------------------------------
        // Up to `burst` Woodcock steps per iteration: a lane keeps stepping through virtual
        // collisions and stops at a real event or the grid boundary.  Each lane draws its
        // own stream in the reference's order, so the burst length changes the schedule,
        // not the histories.
        const int burst = ws.burst; // at least one: every iteration makes progress
        for (int k = 0; k < burst; ++k) {
            if (s.state == FLYING) {
                // a flight drawn with the local majorant ends without a collision test
                // where that majorant stops holding (truncated: drawn again from there)
                const Real flight = -m_log2(up<Real>(s.rng.uniform_open())) * (s.stepK * s.cinv);
                const Real R = m_abs(s.cR);
                const bool truncated = flight > R;
                if (truncated && s.cR < Real(0.0)) {
                    // outside the body box the flight may reach further than the ball:
                    // drawn again once the setup stage has looked how far
                    s.rng.step_back();
                    s.state = REACH;
                } else {
                    const Real step = m_min(flight, R);
                    s.ph.px = m_fma(s.ph.dx, step, s.ph.px);
                    s.ph.py = m_fma(s.ph.dy, step, s.ph.py);
                    s.ph.pz = m_fma(s.ph.dz, step, s.ph.pz);
                    // grid coordinates (p - lo) / spacing as one FMA each, rounded down; the photon
                    // is inside while all three lie in [0, dims) (one unsigned compare each: a
                    // negative or saturated conversion falls outside), which bounds the voxel index
                    const uint32_t ix = static_cast<uint32_t>(m_floor_int(m_fma(s.ph.px, up<Real>(w.inv_spacing[0]), -up<Real>(w.lo_inv[0]))));
                    const uint32_t iy = static_cast<uint32_t>(m_floor_int(m_fma(s.ph.py, up<Real>(w.inv_spacing[1]), -up<Real>(w.lo_inv[1]))));
                    const uint32_t iz = static_cast<uint32_t>(m_floor_int(m_fma(s.ph.pz, up<Real>(w.inv_spacing[2]), -up<Real>(w.lo_inv[2]))));
                    if (!(ix < w.dims[0] && iy < w.dims[1] && iz < w.dims[2])) {
                        s.state = IDLE;
                    } else {
                        ++s.hist_steps;
                        const Real cinv = s.cinv; // the majorant this flight was drawn with
                        // the voxel is read before the majorant cell, so that the two reads
                        // overlap; a truncated flight does not need it (three in ten of the CT
                        // workload's, a read from DRAM each with 8-byte voxels)
                        VoxelRaw<PALETTE> raw {};
                        if constexpr (!LEAN) {
                            s.vidx = voxel_index<PALETTE>(w, ix, iy, iz);
                            if (!truncated)
                                raw = load_voxel<PALETTE>(w, s.vidx);
                        }
                        if (FAST || p.majorant.cells) {
                            const MajorantGrid& g = p.majorant;
                            const uint32_t c = (iz >> g.shift[2]) * g.nxy + (iy >> g.shift[1]) * g.nx + (ix >> g.shift[0]);
                            const float2 cell = __ldg(g.cells + (c * g.bands + s.band));
                            s.cinv = up<Real>(cell.x);
                            s.cR = up<Real>(cell.y);
                        }
                        if (!truncated) {
                            if constexpr (LEAN) {
                                s.vidx = voxel_index<PALETTE>(w, ix, iy, iz);
                                raw = load_voxel<PALETTE>(w, s.vidx);
                            }
                            collide<MODEL, PALETTE, FORCED, FAST>(s, ws, p, L, pal, table, raw, cinv);
                        }
                    }
                }
            }
        }

        // ---- interaction pass -----------------------------------------------------------
        // Every waiting lane runs in one pass once enough of them wait.  Photoelectric,
        // Compton and Rayleigh lanes share the type draw, for LIVERMORE the table quantile
        // (Compton and Rayleigh angles both come from an energy-row table), the azimuth and
        // the rotation; each lane draws from its stream in the order of the reference's
        // samplers.
        const unsigned waiting = __ballot_sync(FULL_MASK, waits_for_event(s.state));
        if (!waiting)
            return;
        if (__popc(waiting) < interact_t && !drain && __any_sync(FULL_MASK, s.state == FLYING || s.state == REACH))
            return;
        bool do_score = false;
        Real deposit = Real(0.0); // energy imparted x weight to score
        bool done = waits_for_event(s.state); // the lane's event ends in this pass
        const bool forced = FORCED && s.state < 0;
        bool photo = false, compton = false;
        Real imparted = Real(0.0), cosA = Real(1.0);
        bool turn = true;
        bool ok = true; // false: a sampling loop hit its cap
        int code = forced ? -s.state : s.state;
        if (done && (MODEL != 2 || code < TRYING)) {
            const int mat = code - 1;
            const Real E = s.ph.energy;
            Real p0, p01;
            if constexpr (SHARES) {
                p0 = s.p0;
                p01 = s.p01;
            } else {
                type_shares(L, m, mat, E, p0, p01);
            }
            const Real r3 = up<Real>(s.rng.uniform());
            photo = !forced && r3 < p0;
            compton = forced ? r3 * (Real(1.0) - p0) < p01 - p0 : (!photo && r3 < p01);
            if constexpr (MODEL == 1) {
                if (photo) {
                    imparted = E;
                    s.ph.energy = Real(0.0);
                    turn = false;
                } else {
                    Real fe;
                    // in double the logarithm of the setup serves again
                    const int row = table_row(m, SHARES ? s.logE * Real(2.30258509299404568402) : m_log(E), fe);
                    const float* tab = p.lut + (compton ? m.off_csf : m.off_ray) + (mat * m.tab_ne + row) * (m.tab_nu + 1);
                    const Real x = table_quantile(tab, m.tab_nu, up<Real>(s.rng.uniform()), fe);
                    if (compton) {
                        Real e;
                        compton_from_fraction(E, x, e, cosA);
                        s.ph.energy = E * e;
                        imparted = E - s.ph.energy;
                    } else {
                        cosA = Real(1.0) - Real(2.0) * x; // q^2 / q_max^2 = (1 - cos) / 2
                    }
                }
            } else if constexpr (MODEL == 0) {
                if (photo)
                    imparted = photo_sample<MODEL>(L, m, s.ph.energy, mat, s.rng, cosA, turn);
                else if (compton)
                    ok = compton_sample<MODEL>(L, p.lut, m, s.ph.energy, mat, s.rng, cosA, imparted, turn);
                else
                    ok = rayleigh_sample<MODEL>(p.lut, m, E, mat, s.rng, cosA);
            } else {
                if (photo) {
                    imparted = photo_sample<MODEL>(L, m, s.ph.energy, mat, s.rng, cosA, turn);
                } else if (!compton) {
                    ok = rayleigh_sample<MODEL>(p.lut, m, E, mat, s.rng, cosA);
                } else {
                    const int shell = compton_shell(L, m, E, mat, s.rng);
                    if (shell < 0)
                        turn = false; // rejected: nothing changes, zero energy imparted
                    else
                        code = TRYING | (mat * N_SHELLS + shell);
                }
            }
        }
        if constexpr (MODEL == 2) {
            // The rejection draws (compton_ia) of all lanes with a shell: the energy draws
            // repeat while enough lanes are rejected, then the accepted ones draw the shift.
            // Lanes that looped until each was accepted left the warp with 7.4 of them on
            // average.
            bool trying = done && code >= TRYING;
            done = done && !trying;
            while (true) {
                bool energy_ok = false;
                Real e = Real(0.0), t = Real(0.0);
                while (true) {
                    if (trying && !energy_ok && (code >> TRY_SHIFT) < REJECTION_CAP) {
                        energy_ok = compton_ia_energy(s.ph.energy, s.rng, e, t);
                        code += 1 << TRY_SHIFT;
                    }
                    if (__popc(__ballot_sync(FULL_MASK, trying && !energy_ok && (code >> TRY_SHIFT) < REJECTION_CAP)) < MIN_TRYING)
                        break;
                }
                if (trying) {
                    if (energy_ok && compton_ia_shift(L + m.off_shells + (code & (TRYING - 1)) * SHELL_FLOATS, s.ph.energy, s.rng, t, e, cosA)) {
                        const Real E = s.ph.energy;
                        s.ph.energy = E * e;
                        imparted = E - s.ph.energy;
                        trying = false;
                    } else if ((code >> TRY_SHIFT) >= REJECTION_CAP) {
                        ok = false;
                        trying = false;
                    }
                    compton = done = !trying;
                }
                if (__popc(__ballot_sync(FULL_MASK, trying)) < MIN_ROUND)
                    break;
            }
            if (trying)
                s.state = forced ? -code : code;
        }
        if (done) {
            s.state = FLYING;
            if (turn && ok) {
                Real sin_phi, cos_phi;
                rng_azimuth(s.rng, &sin_phi, &cos_phi);
                peturb(s.ph.dx, s.ph.dy, s.ph.dz, cosA, sin_phi, cos_phi, !FAST && p.normalize_direction);
            }
            if (!ok) {
                atomicAdd(&ws.overflows, 1u);
                s.state = IDLE;
            } else if (photo || compton) {
                do_score = true;
                if (s.ph.energy < Real(ENERGY_CUTOFF_D)) {
                    deposit = add_rounded(imparted, s.ph.energy) * s.ph.weight;
                    s.ph.energy = Real(0.0);
                    s.state = IDLE;
                } else {
                    deposit = imparted * s.ph.weight;
                    s.state = SETUP;
                }
            }
            if (s.state != IDLE) {
                if (forced)
                    s.ph.weight *= (Real(1.0) - s.forced_wc);
                roulette(s);
            }
            if (do_score && !isfinite(deposit)) {
                // never let a non-finite value into the FP64 accumulators: end the
                // history and report it through the overflow counter
                do_score = false;
                s.state = IDLE;
                atomicAdd(&ws.overflows, 1u);
            }
        }
        // ---- scoring; the warp is converged here ----------------------------------------
        if (!FAST && p.tally_mode == 2) {
            const unsigned scoring = __ballot_sync(FULL_MASK, do_score);
            if (do_score)
                score_aggregated(p, scoring, s.vidx, deposit);
        } else if (do_score) {
            score<FAST>(p, s.vidx, deposit);
        }
        if (do_score)
            atomicAdd(&ws.deposits, 1u);
    }

    // Counts the steps of the photons a warp's lanes finished (before they are
    // refilled or at a flush).  Called by all 32 lanes.
    template <class Real, class Index>
    __device__ __forceinline__ void count_steps(LaneT<Real, Index>& s, WarpState& ws, bool finished)
    {
        const unsigned n = __reduce_add_sync(FULL_MASK, finished ? s.hist_steps : 0u);
        if ((threadIdx.x & 31) == 0)
            ws.steps += n;
        if (finished)
            s.hist_steps = 0;
    }

    // Adds the warp's counters to a job's counters, the steps of photons in flight
    // included, and clears them.  Called by all 32 lanes.
    template <class Real, class Index>
    __device__ __forceinline__ void flush_counters(LaneT<Real, Index>& s, WarpState& ws, JobCounters* c)
    {
        count_steps(s, ws, true); // counted once: the photons' steps so far
        add_counters(ws, c);
    }

    // ---- single-job transport kernel ----------------------------------------------------
    //
    // Warp-synchronous loop, bound by instruction issue at about half of a warp's lanes:
    // what a stage costs is paid by the warp whatever its lanes, so each stage runs when
    // enough lanes want it.  Idle lanes take photons from the warp's pool, which all 32
    // lanes fill together; new photons and new energies are set up together; the lanes
    // then fly a burst; and once enough of them wait for an event the interactions run in
    // one pass.  Four blocks per SM, of 288 threads where 56 registers are enough and of 256
    // with 64 (see transport_block; 48 or 40 registers spilled and ran 20 to 30 % slower);
    // what belongs to the warp lives in shared memory, the LUT too (read through L1: CT 8 %,
    // DX 12 %, IA 4 % slower).  Against photons sampled in place, the box test and the
    // attenuation in the flight loop and a vote after each flight, kernel alone: CT
    // 512 x 512 x 200 of 1e8 histories 13.4 -> 11.4 ms, DX 160^3 of 5e6 0.753 -> 0.549 ms,
    // with impulse approximation (127^3, 4e6) 1.85 -> 1.13 ms, CTDI phantom of 1e7 with
    // forced scoring 1.29 -> 1.01 ms, DX 96^3 of 1e6 in FP64 6.4 -> 4.3 ms (two blocks per
    // SM: about twice the registers; FP64 pipe 86 % busy).
    template <class Real, int MODEL, bool PALETTE, bool FORCED, bool FAST>
    __global__ void __launch_bounds__(transport_block(FAST, FORCED, PALETTE, MODEL), sizeof(Real) == 4 ? DXMC_MIN_BLOCKS_PER_SM : 2) transport_kernel(const __grid_constant__ TransportParams p)
    {
        extern __shared__ float4 smem_f4[];
        // a job cancelled before its kernel ran takes no history (the read over the link
        // overlaps the staging below)
        __shared__ int cancelled;
        const int flag = threadIdx.x == 0 && p.cancel ? *p.cancel : 0;
        // in the fast kernels a shared-memory address to the compiler (32-bit loads)
        const float* L = FAST ? reinterpret_cast<const float*>(smem_f4) : p.lut;
        size_t smem_off = 0;
        if (FAST || p.lut_in_smem) {
            float4* dst = smem_f4;
            const float4* src = reinterpret_cast<const float4*>(p.lut);
            const int n4 = ((MODEL == 2 ? p.lut_meta.total_floats : p.lut_meta.off_shells) + 3) / 4;
            for (int i = threadIdx.x; i < n4; i += blockDim.x)
                dst[i] = __ldg(src + i);
            if constexpr (!FAST)
                L = reinterpret_cast<const float*>(smem_f4);
            smem_off = static_cast<size_t>(n4);
        }
        const PaletteEntry* pal = nullptr;
        if constexpr (PALETTE) {
            PaletteEntry* spal = reinterpret_cast<PaletteEntry*>(smem_f4 + smem_off);
            for (int i = threadIdx.x; i < PALETTE_MAX; i += blockDim.x)
                spal[i] = i < p.world.palette_n ? p.world.palette[i] : PaletteEntry { Real(0.0), 0u };
            pal = spal;
            smem_off += PALETTE_MAX * sizeof(PaletteEntry) / sizeof(float4);
        }
        float* table = nullptr; // this lane's column of the attenuation table
        if constexpr (FAST)
            table = reinterpret_cast<float*>(smem_f4 + smem_off) + threadIdx.x;
        if (threadIdx.x == 0)
            cancelled = flag;
        __syncthreads();
        const int lane = threadIdx.x & 31;
        const unsigned lanemask_lt = (1u << lane) - 1u;
        const int regen_t = p.regen_threshold;
        const int interact_t = p.interact_threshold;
        const bool use_queue = !FAST && p.queue.pos_energy != nullptr;
        const uint64_t source_total = use_queue ? p.counters->queue_count : p.total_histories;

        constexpr int WARPS = transport_block(FAST, FORCED, PALETTE, MODEL) / 32;
        __shared__ WarpState states[WARPS];
        __shared__ PhotonPool<Real> pools[WARPS];
        WarpState& ws = states[threadIdx.x >> 5];
        PhotonPool<Real>& pool = pools[threadIdx.x >> 5];
        if (lane == 0) {
            ws = WarpState {};
            const uint64_t unit = static_cast<uint64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
            ws.next = work_unit(p.work, unit, ws.end);
            if (cancelled) {
                ws.next = source_total;
                ws.end = ~0ull; // and no further unit
            }
            ws.burst = p.woodcock_burst > 0 ? p.woodcock_burst : (sizeof(Real) == 8 ? SHORT_BURST : START_BURST);
        }
        __syncwarp();
        LaneT<Real, typename VoxelRaw<PALETTE>::Index> s {};
        s.state = IDLE;
        bool exhausted = false; // no photon left to take

        while (true) {
            // ---- refill idle lanes together ------------------------------------------------
            unsigned need = __ballot_sync(FULL_MASK, s.state == IDLE);
            if (!exhausted && __popc(need) >= regen_t) {
                while (need) {
                    const int pooled = ws.pooled;
                    if (pooled == 0) {
                        // a unit of the job is done: the job's progress, and the next unit
                        if (ws.next >= ws.end && (ws.histories >= PUBLISH_HISTORIES || ws.steps >= CARRY))
                            add_counters(ws, p.counters);
                        const uint64_t warps = static_cast<uint64_t>(gridDim.x) * (blockDim.x >> 5);
                        DeviceWarp self;
                        const uint64_t next = next_ids(self, ws, p.work, warps, use_queue ? &p.counters->next_photon : &p.counters->next_history,
                            source_total, [&p] { return p.cancel && *p.cancel; });
                        if (next >= source_total) {
                            exhausted = true;
                            break;
                        }
                        // all lanes sample the next 32 ids; those inside the grid go into the pool
                        const bool mine = next + lane < source_total;
                        bool inside = false;
                        PhotonT<Real> ph {};
                        Rng rng {};
                        if (mine) {
                            if (use_queue) {
                                load_queued(ph, rng, p.queue, next + lane);
                                inside = true;
                            } else {
                                inside = sample_history(ph, rng, p, next + lane);
                            }
                        }
                        const unsigned sampled = __ballot_sync(FULL_MASK, mine);
                        const unsigned entered = __ballot_sync(FULL_MASK, inside);
                        if (inside)
                            pool.put(__popc(entered & lanemask_lt), ph, rng);
                        if (lane == 0) {
                            ws.next = next + 32;
                            ws.pooled = __popc(entered);
                            if (!use_queue)
                                ws.histories += __popc(sampled);
                            // the photons in flight are counted as histories, not yet by their steps: 64 of
                            // 4096 at most, but wait for a few hundred steps
                            if (p.woodcock_burst == 0 && ws.steps >= 256)
                                ws.burst = (ws.deposits + ws.forced_deposits + ws.histories) * 100 > ws.steps * LONG_BURST_STOPS ? SHORT_BURST : LONG_BURST;
                        }
                        __syncwarp();
                        continue;
                    }
                    const int rank = __popc(need & lanemask_lt);
                    const bool mine = ((need >> lane) & 1u) && rank < pooled;
                    const unsigned taken = __ballot_sync(FULL_MASK, mine);
                    count_steps(s, ws, mine);
                    if (mine) {
                        pool.get(pooled - 1 - rank, s.ph, s.rng);
                        s.start_photon();
                    }
                    if (lane == 0)
                        ws.pooled = pooled - __popc(taken);
                    need &= ~taken;
                    __syncwarp(); // the pool may be filled again
                }
            }
            if (exhausted && __ballot_sync(FULL_MASK, s.state != IDLE) == 0u)
                break;
            advance<MODEL, PALETTE, FORCED, FAST>(s, ws, p, L, pal, table, exhausted, interact_t);
        }
        flush_counters(s, ws, p.counters);
    }

    // ---- batched transport kernel ------------------------------------------------------
    //
    // Many jobs (worlds, LUTs, sources, tallies of their own) in one persistent launch.
    // A block works on one job at a time: its warps take chunks of histories from the
    // job's own counter until none is left, finish their photons, and the block goes on
    // to the next job that has histories.  Blocks start spread over the jobs by their
    // histories, so most never change more than once or twice.  Each history keeps its
    // own random stream, so a job's tallies do not depend on what else runs in the batch.
    //
    // Bound by the latency of voxel, grid and LUT reads through L1, so what counts is L1
    // capacity: the job's parameters and palette lie in shared memory once per block (3 KB;
    // once per warp took 22 KB and let the warps of a block read the tables of several
    // jobs), and the tables stay in global memory.  Twenty DX jobs of 1.5e5 to 1.1e6
    // histories: items of 525 histories from one queue, a job per warp, 1.81 ms; this
    // 1.57 ms; the LUT in shared memory besides 1.62, a pool of sampled photons per warp
    // besides 1.80.  Sixteen DX jobs of 5e6 on average: 9.5 -> 8.3 ms.
    constexpr int BATCH_WARPS = 8; // 256-thread blocks

    template <int MODEL>
    __global__ void __launch_bounds__(32 * BATCH_WARPS, DXMC_MIN_BLOCKS_PER_SM) batch_transport_kernel(const __grid_constant__ BatchParams b)
    {
        __shared__ TransportParams p;
        __shared__ PaletteEntry pal[PALETTE_MAX];
        __shared__ WarpState states[BATCH_WARPS];
        __shared__ uint32_t chosen;
        const int lane = threadIdx.x & 31;
        const int warp = threadIdx.x >> 5;
        const unsigned lanemask_lt = (1u << lane) - 1u;
        const BatchControl* ctl = b.control;
        const BatchItem* items = b.items + ctl->item_base[MODEL];
        const uint32_t n_items = static_cast<uint32_t>(ctl->n_items[MODEL]);
        const uint64_t chunk = ctl->chunk;
        const int regen_t = ctl->regen_threshold;
        const int interact_t = ctl->interact_threshold;
        WarpState& ws = states[warp];
        if (lane == 0)
            ws = WarpState {};
        __syncwarp();
        LaneT<float, uint64_t> s {};
        s.state = IDLE;

        // the block starts at its share of the jobs' histories laid end to end
        uint32_t at = 0;
        {
            const uint64_t position = ctl->histories[MODEL] / gridDim.x * blockIdx.x;
            uint32_t above = n_items; // the last job that starts at or before it
            while (above - at > 1) {
                const uint32_t mid = (at + above) / 2;
                if (items[mid].first <= position)
                    at = mid;
                else
                    above = mid;
            }
        }
        while (true) {
            // ---- the block's next job: the first from `at` on with histories left ------------
            if (warp == 0) {
                uint32_t seen = 0;
                unsigned found = 0;
                while (seen < n_items) {
                    uint32_t c = at + lane;
                    c = c < n_items ? c : (c - n_items) % n_items;
                    const bool some = seen + lane < n_items
                        && *reinterpret_cast<const volatile unsigned long long*>(&items[c].counters->next_history) < items[c].histories;
                    found = __ballot_sync(FULL_MASK, some);
                    if (found) {
                        at = __shfl_sync(FULL_MASK, c, __ffs(found) - 1);
                        break;
                    }
                    at = at + 32 < n_items ? at + 32 : (at + 32 - n_items) % n_items;
                    seen += 32;
                }
                if (lane == 0)
                    chosen = found ? at : n_items;
            }
            __syncthreads();
            at = chosen;
            if (at >= n_items)
                break;
            {
                const int* src = reinterpret_cast<const int*>(b.jobs + items[at].job);
                int* dst = reinterpret_cast<int*>(&p);
                for (int k = threadIdx.x; k < static_cast<int>(sizeof(TransportParams) / sizeof(int)); k += blockDim.x)
                    dst[k] = __ldg(src + k);
            }
            __syncthreads();
            const int np = p.world.palette_index ? p.world.palette_n : 0;
            for (int k = threadIdx.x; k < PALETTE_MAX; k += blockDim.x)
                pal[k] = k < np ? p.world.palette[k] : PaletteEntry { 0.0f, 0u };
            if (lane == 0)
                ws.burst = p.woodcock_burst > 0 ? p.woodcock_burst : START_BURST;
            __syncthreads();

            // ---- its histories, a chunk at a time ----------------------------------------------
            const uint64_t histories = items[at].histories;
            uint64_t next = 0, end = 0;
            bool exhausted = false;
            while (true) {
                unsigned need = __ballot_sync(FULL_MASK, s.state == IDLE && !exhausted);
                if (need && __popc(need) >= regen_t) {
                    while (need) {
                        if (next >= end) {
                            unsigned long long first = 0;
                            if (lane == 0) {
                                first = atomicAdd(&p.counters->next_history, static_cast<unsigned long long>(chunk));
                                carry_counters(ws);
                            }
                            next = __shfl_sync(FULL_MASK, first, 0);
                            end = min(next + chunk, histories);
                            if (next >= end) {
                                exhausted = true;
                                break;
                            }
                        }
                        const uint64_t avail = end - next;
                        const unsigned rank = __popc(need & lanemask_lt);
                        const bool mine = ((need >> lane) & 1u) && rank < avail;
                        const unsigned taken = __ballot_sync(FULL_MASK, mine);
                        count_steps(s, ws, mine);
                        if (lane == 0) {
                            ws.histories += __popc(taken);
                            if (p.woodcock_burst == 0 && ws.steps >= 256)
                                ws.burst = (ws.deposits + ws.forced_deposits + ws.histories) * 100 > ws.steps * LONG_BURST_STOPS ? SHORT_BURST : LONG_BURST;
                        }
                        __syncwarp(); // the other lanes read the burst next
                        if (mine)
                            take_history(s, p, next + rank);
                        next += __popc(taken);
                        need &= ~taken;
                    }
                }
                if (exhausted && __ballot_sync(FULL_MASK, s.state != IDLE) == 0u)
                    break;
                if (p.world.palette_index)
                    advance<MODEL, true, true, false, true>(s, ws, p, p.lut, pal, nullptr, exhausted, interact_t);
                else
                    advance<MODEL, false, true, false, true>(s, ws, p, p.lut, pal, nullptr, exhausted, interact_t);
            }
            flush_counters(s, ws, p.counters);
            __syncthreads(); // the job's parameters and tables are read no more
        }
    }

    // ---- photon generation pass ---------------------------------------------------------
    // One thread per history: Exposure::sampleParticle + transportParticleToWorld with
    // every lane of the warp busy; photons inside the world are appended to the queue
    // together with the state of their random stream.
    __global__ void __launch_bounds__(256) generate_kernel(const __grid_constant__ TransportParams p, uint64_t first, uint64_t count)
    {
        const int lane = threadIdx.x & 31;
        unsigned long long generated = 0;
        for (uint64_t base = blockIdx.x * static_cast<uint64_t>(blockDim.x); base < count; base += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
            const uint64_t i = base + threadIdx.x;
            bool inworld = false;
            PhotonT<float> ph {};
            Rng rng;
            if (i < count) {
                inworld = sample_history(ph, rng, p, first + i);
                ++generated;
            }
            const unsigned mask = __ballot_sync(FULL_MASK, inworld);
            unsigned long long slot0 = 0;
            if (lane == 0 && mask)
                slot0 = atomicAdd(&p.counters->queue_count, static_cast<unsigned long long>(__popc(mask)));
            slot0 = __shfl_sync(FULL_MASK, slot0, 0);
            if (inworld) {
                const uint64_t q = slot0 + __popc(mask & ((1u << lane) - 1u));
                p.queue.pos_energy[q] = make_float4(ph.px, ph.py, ph.pz, ph.energy);
                p.queue.dir_weight[q] = make_float4(ph.dx, ph.dy, ph.dz, ph.weight);
                p.queue.rng[q] = make_uint4(rng.s0, rng.s1, rng.s2, rng.s3);
            }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
            generated += __shfl_down_sync(FULL_MASK, generated, off);
        if (lane == 0 && generated)
            atomicAdd(&p.counters->histories_done, generated);
    }

    // ---- post-processing (transport.hpp:780-816) -------------------------------------
    template <typename TallyT>
    __global__ void postprocess_kernel(const TallyT* __restrict__ tally, const Voxel* __restrict__ voxels,
        const uint8_t* __restrict__ palette_index, const PaletteEntry* __restrict__ palette, uint64_t n, int mode,
        double histories, double voxel_volume_cm3, double calibration, double* __restrict__ dose, double* __restrict__ variance,
        const uint32_t* __restrict__ counts, uint32_t* __restrict__ counts_out)
    {
        const double h_inv = 1.0 / (histories - 1.0);
        const double h_d = 1.0e3 / histories;
        const double h_v = 1.0e6 / histories;
        for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n; i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
            const double e = static_cast<double>(tally[2 * i]);
            const double ee = static_cast<double>(tally[2 * i + 1]);
            double d = e, v = ee;
            if (mode == 1) { // EV_PER_HISTORY: normalizeScoring
                d = e * h_d;
                v = (ee * h_v - d * d) * h_inv;
            } else if (mode == 2) { // DOSE: energyImpartedToDose
                const double de = static_cast<double>(voxels ? voxels[i].density : palette[palette_index[i]].density);
                const double mass = de * voxel_volume_cm3 * 0.001;
                const double f = calibration / mass;
                d = de > 0.0 ? e * f : 0.0;
                v = de > 0.0 ? ee * f * f : 0.0;
            }
            if (dose)
                dose[i] = d;
            if (variance)
                variance[i] = v;
            if (counts_out)
                counts_out[i] = __ldg(counts + i);
        }
    }

    // Copies 1 .. copies - 1 of the records added to copy 0, in that order.
    __global__ void fold_tallies_kernel(TallyRecord* __restrict__ rec, const TallyRecord* __restrict__ more, uint64_t n, uint32_t copies)
    {
        for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n; i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
            uint32_t events = 0;
            double e = 0.0, ee = 0.0;
            for (uint32_t c = 1; c < copies; ++c) {
                const TallyRecord r = more[(c - 1) * n + i];
                events += r.events;
                e += r.energy;
                ee += r.energy2;
            }
            if (events) {
                rec[i].energy += e;
                rec[i].energy2 += ee;
                rec[i].events += events;
            }
        }
    }

    // Post-processing from tally records: one 32-byte record read per voxel; the
    // results in double (Result<double>) or float (Result<float>), computed in double.
    template <typename OutT>
    __global__ void postprocess_records_kernel(const TallyRecord* __restrict__ rec, const Voxel* __restrict__ voxels,
        const uint8_t* __restrict__ palette_index, const PaletteEntry* __restrict__ palette, uint64_t n, int mode,
        double histories, double voxel_volume_cm3, double calibration, OutT* __restrict__ dose, OutT* __restrict__ variance,
        uint32_t* __restrict__ counts_out, const JobCounters* counters, JobCounters* counters_out)
    {
        if (counters_out && blockIdx.x == 0 && threadIdx.x == 0)
            *counters_out = *counters; // the job has ended; saves a copy of its own
        const double h_inv = 1.0 / (histories - 1.0);
        const double h_d = 1.0e3 / histories;
        const double h_v = 1.0e6 / histories;
        for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n; i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
            const double2 ee2 = __ldcs(reinterpret_cast<const double2*>(rec + i));
            const double e = ee2.x, ee = ee2.y;
            double d = e, v = ee;
            if (mode == 1) { // EV_PER_HISTORY: normalizeScoring
                d = e * h_d;
                v = (ee * h_v - d * d) * h_inv;
            } else if (mode == 2) { // DOSE: energyImpartedToDose
                const double de = static_cast<double>(voxels ? voxels[i].density : palette[palette_index[i]].density);
                const double mass = de * voxel_volume_cm3 * 0.001;
                const double f = calibration / mass;
                d = de > 0.0 ? e * f : 0.0;
                v = de > 0.0 ? ee * f * f : 0.0;
            }
            if (dose)
                dose[i] = static_cast<OutT>(d);
            if (variance)
                variance[i] = static_cast<OutT>(v);
            if (counts_out)
                counts_out[i] = __ldcs(&rec[i].events);
        }
    }

    // ---- per-material maximum density (attenuationinterpolator.hpp:48-60) ------------
    __global__ void max_density_kernel(const Voxel* __restrict__ voxels, uint64_t n, unsigned int* out_bits, int n_materials)
    {
        extern __shared__ unsigned int sbits[];
        for (int i = threadIdx.x; i < n_materials; i += blockDim.x)
            sbits[i] = 0u;
        __syncthreads();
        for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n; i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
            const uint2 raw = __ldg(reinterpret_cast<const uint2*>(voxels) + i);
            const int mat = raw.y & 0xffu;
            const float d = __uint_as_float(raw.x);
            if (mat < n_materials && d > 0.0f)
                atomicMax(&sbits[mat], raw.x); // non-negative floats order like their bits
        }
        __syncthreads();
        for (int i = threadIdx.x; i < n_materials; i += blockDim.x)
            if (sbits[i])
                atomicMax(out_bits + i, sbits[i]);
    }

    // ---- probes ------------------------------------------------------------------------
    __global__ void probe_lut_kernel(const float* L, LutMeta m, int material, const double* energies, int n, double* out_att, double* out_maxinv)
    {
        const int i = blockIdx.x * blockDim.x + threadIdx.x;
        if (i >= n)
            return;
        const float E = static_cast<float>(energies[i]);
        const float logE = __log10f(E);
        const int seg = lut_segment(L, m, logE);
        float a, b, c;
        lut_attenuation(L, m, material, logE, seg, a, b, c);
        out_att[3 * i] = a;
        out_att[3 * i + 1] = b;
        out_att[3 * i + 2] = c;
        out_maxinv[i] = lut_max_inverse(L, m, logE, seg);
    }

    template <int MODEL>
    __global__ void probe_interactions_kernel(const float* L, LutMeta m, int material, int kind, float energy, uint64_t n, uint64_t seed,
        float* out_cos, float* out_energy, float* out_dep)
    {
        for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n; i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
            Rng rng;
            rng.init(seed, i);
            PhotonT<float> ph { 0, 0, 0, 0, 0, 1, energy, 1 };
            float dep = 0.0f;
            bool ok = true;
            float cosA = 1.0f;
            bool turn = true;
            if (kind == 0)
                dep = photo_sample<MODEL>(L, m, ph.energy, material, rng, cosA, turn);
            else if (kind == 1)
                ok = compton_sample<MODEL>(L, L, m, ph.energy, material, rng, cosA, dep, turn);
            else
                ok = rayleigh_sample<MODEL>(L, m, ph.energy, material, rng, cosA);
            if (turn && ok) {
                float sin_phi, cos_phi;
                rng_azimuth(rng, &sin_phi, &cos_phi);
                peturb(ph.dx, ph.dy, ph.dz, cosA, sin_phi, cos_phi);
            }
            const float len = sqrtf(ph.dx * ph.dx + ph.dy * ph.dy + ph.dz * ph.dz);
            out_cos[i] = ok ? (len > 0 ? ph.dz / len : 1.0f) : 2.0f;
            out_energy[i] = ph.energy;
            out_dep[i] = dep;
        }
    }

    // Histogram of the per-history streams' output (the generator every sampler
    // draws from): n_streams streams of `draws` values each.  kind 0: uniform()
    // in [0, 1); kind 1: uniform_open() in (0, 1], binned as 1 - u; kind 2:
    // below(nbins).  hist[nbins] counts values outside their stated range.
    __global__ void probe_uniform_kernel(uint64_t seed, uint64_t n_streams, uint32_t draws, int kind, int nbins,
        unsigned long long* hist)
    {
        extern __shared__ unsigned int sbins[];
        for (int i = threadIdx.x; i <= nbins; i += blockDim.x)
            sbins[i] = 0u;
        __syncthreads();
        for (uint64_t h = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; h < n_streams;
             h += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
            Rng rng;
            rng.init(seed, h);
            for (uint32_t k = 0; k < draws; ++k) {
                int b;
                if (kind == 0) {
                    const float u = rng.uniform();
                    b = (u >= 0.0f && u < 1.0f) ? min(static_cast<int>(u * nbins), nbins - 1) : nbins;
                } else if (kind == 1) {
                    const float u = rng.uniform_open();
                    b = (u > 0.0f && u <= 1.0f) ? min(static_cast<int>((1.0f - u) * nbins), nbins - 1) : nbins;
                } else {
                    const uint32_t v = rng.below(static_cast<uint32_t>(nbins));
                    b = v < static_cast<uint32_t>(nbins) ? static_cast<int>(v) : nbins;
                }
                atomicAdd(&sbins[b], 1u);
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i <= nbins; i += blockDim.x)
            if (sbins[i])
                atomicAdd(hist + i, static_cast<unsigned long long>(sbins[i]));
    }

} // namespace

// The kernel of a job: one for the options of nearly every job (TransportVariant::fast),
// without the forced-scoring code where the world has no measurement map, and one for
// all others.
template <class Real, int MODEL, bool PALETTE>
static void* transport_entry(bool forced, bool fast)
{
    if constexpr (sizeof(Real) == 4) {
        if (fast)
            return forced ? reinterpret_cast<void*>(&transport_kernel<Real, MODEL, PALETTE, true, true>)
                          : reinterpret_cast<void*>(&transport_kernel<Real, MODEL, PALETTE, false, true>);
    }
    return reinterpret_cast<void*>(&transport_kernel<Real, MODEL, PALETTE, true, false>);
}

template <class Real>
static void* transport_function_as(int model, bool palette, bool forced, bool fast)
{
    if (palette)
        return model == 0 ? transport_entry<Real, 0, true>(forced, fast)
                          : (model == 1 ? transport_entry<Real, 1, true>(forced, fast) : transport_entry<Real, 2, true>(forced, fast));
    return model == 0 ? transport_entry<Real, 0, false>(forced, fast)
                      : (model == 1 ? transport_entry<Real, 1, false>(forced, fast) : transport_entry<Real, 2, false>(forced, fast));
}

static void* transport_function(const TransportVariant& v)
{
    return v.precision == 1 ? transport_function_as<double>(v.model, v.palette, true, false)
                            : transport_function_as<float>(v.model, v.palette, v.forced, v.fast);
}

TransportVariant transport_variant(const TransportParams& p, int model, bool queued)
{
    TransportVariant v;
    v.model = model;
    v.precision = p.precision;
    v.palette = p.world.palette_index != nullptr;
    v.forced = p.world.has_measurement != 0;
    v.fast = p.precision != 1 && p.lut_meta.n_materials <= ATT_TABLE_MATERIALS && p.lut_in_smem && p.majorant.cells && p.records && p.tally_mode == 0
        && !p.normalize_direction && !queued;
    if (v.fast) {
        const size_t most = model == 2 ? FAST_SHARED_BYTES_IA : FAST_SHARED_BYTES;
        const auto resident = [&](bool fast) { // shared memory of an SM's blocks
            constexpr size_t PER_WARP = sizeof(WarpState) + sizeof(PhotonPool<float>), RESERVED = 1024;
            TransportVariant u = v;
            u.fast = fast;
            const int warps = transport_block(fast, v.forced, v.palette, model) / 32;
            return DXMC_MIN_BLOCKS_PER_SM * (transport_smem_bytes(u, p.lut_meta, true) + warps * PER_WARP + RESERVED);
        };
        v.fast = resident(true) <= most || (v.forced && resident(false) > most);
    }
    return v;
}

const void* batch_kernel_function(int model)
{
    if (model == 0)
        return reinterpret_cast<const void*>(&batch_transport_kernel<0>);
    if (model == 1)
        return reinterpret_cast<const void*>(&batch_transport_kernel<1>);
    return reinterpret_cast<const void*>(&batch_transport_kernel<2>);
}

int batch_max_blocks_per_sm(int model)
{
    int n = 0;
    cudaError_t e;
    if (model == 0)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, batch_transport_kernel<0>, 256, 0);
    else if (model == 1)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, batch_transport_kernel<1>, 256, 0);
    else
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, batch_transport_kernel<2>, 256, 0);
    return e == cudaSuccess ? n : 0;
}

cudaError_t launch_generate(const TransportParams& p, uint64_t first, uint64_t count, int grid, cudaStream_t stream)
{
    generate_kernel<<<grid, 256, 0, stream>>>(p, first, count);
    return cudaGetLastError();
}

size_t transport_smem_bytes(const TransportVariant& v, const LutMeta& meta, bool lut_in_smem)
{
    size_t b = lut_in_smem ? (static_cast<size_t>(staged_lut_floats(meta, v.model)) * sizeof(float) + 15) / 16 * 16 : 0;
    if (v.palette)
        b += PALETTE_MAX * sizeof(PaletteEntry);
    if (v.fast)
        b += static_cast<size_t>(meta.n_materials) * ATT_TABLE_LANES * sizeof(float);
    return b;
}

WorkSplit transport_work_split(uint64_t histories, uint64_t warps, bool queued)
{
    WorkSplit w;
    if (queued || warps == 0) { // how many photons wait is known on the device only
        w.large_units = ~0ull >> 16;
        return w;
    }
    const uint64_t rounds = (histories + warps * 32 - 1) / (warps * 32);
    if (rounds <= 2) {
        w.large_units = 0;
    } else if (rounds <= 24) {
        w.large = static_cast<uint32_t>(rounds * 3 / 4) * 32;
        w.large_units = std::min(warps, histories / w.large);
    } else {
        const uint64_t tail = warps * 32 * 6;
        w.large_units = (histories - tail) / w.large;
        w.small = 64;
    }
    return w;
}

cudaError_t launch_transport(const TransportParams& p, int model, int grid, int block, size_t smem, cudaStream_t stream)
{
    void* fn = transport_function(transport_variant(p, model, p.queue.pos_energy != nullptr));
    void* args[] = { const_cast<TransportParams*>(&p) };
    return cudaLaunchKernel(fn, dim3(grid), dim3(block), args, smem, stream);
}

cudaError_t preload_transport_kernels()
{
    for (int model = 0; model < 3; ++model)
        for (int palette = 0; palette < 2; ++palette)
            for (int kind = 0; kind < 4; ++kind) { // FP64; FP32 general, fast, fast with forced scoring
                const TransportVariant v { model, kind == 0 ? 1 : 0, palette != 0, kind != 2, kind >= 2 };
                cudaFuncAttributes attr {};
                const cudaError_t e = cudaFuncGetAttributes(&attr, transport_function(v));
                if (e != cudaSuccess)
                    return e;
            }
    return cudaSuccess;
}

int transport_max_blocks_per_sm(const TransportVariant& v, int block, size_t smem)
{
    void* fn = transport_function(v);
    // The dynamic shared-memory limit is a property of the function, read when a
    // launch (or a graph holding it) is made: it only ever grows, so launches
    // queued or captured earlier with larger LUTs stay valid.
    static std::mutex m;
    static std::unordered_map<void*, int> limit;
    {
        std::lock_guard<std::mutex> lock(m);
        int& cur = limit[fn];
        if (static_cast<int>(smem) > cur) {
            if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) == cudaSuccess)
                cur = static_cast<int>(smem);
        }
    }
    int n = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, block, smem);
    return e == cudaSuccess ? n : 0;
}

cudaError_t launch_postprocess(const double* tally, const WorldParams& w, uint64_t n, int mode, double histories,
    double voxel_volume_cm3, double calibration, double* dose, double* variance, const uint32_t* counts, uint32_t* counts_out,
    cudaStream_t stream)
{
    const int block = 256;
    const int grid = static_cast<int>(std::min<uint64_t>((n + block - 1) / block, 152ull * 16));
    postprocess_kernel<double><<<grid, block, 0, stream>>>(tally, w.palette_index ? nullptr : w.voxels, w.palette_index, w.palette, n, mode,
        histories, voxel_volume_cm3, calibration, dose, variance, counts, counts_out);
    return cudaGetLastError();
}

cudaError_t launch_fold_tallies(TallyRecord* records, const TallyRecord* more, uint64_t n, uint32_t copies, cudaStream_t stream)
{
    const int block = 256;
    const int grid = static_cast<int>(std::min<uint64_t>((n + block - 1) / block, 152ull * 8));
    fold_tallies_kernel<<<grid, block, 0, stream>>>(records, more, n, copies);
    return cudaGetLastError();
}

cudaError_t launch_postprocess_records(const TallyRecord* records, const WorldParams& w, uint64_t n, int mode,
    double histories, double voxel_volume_cm3, double calibration, double* dose, double* variance, uint32_t* counts_out,
    const JobCounters* counters, JobCounters* counters_out, cudaStream_t stream)
{
    const int block = 256;
    const int grid = static_cast<int>(std::min<uint64_t>((n + block - 1) / block, 152ull * 16));
    postprocess_records_kernel<double><<<grid, block, 0, stream>>>(records, w.palette_index ? nullptr : w.voxels, w.palette_index,
        w.palette, n, mode, histories, voxel_volume_cm3, calibration, dose, variance, counts_out, counters, counters_out);
    return cudaGetLastError();
}

cudaError_t launch_postprocess_records_f32(const TallyRecord* records, const WorldParams& w, uint64_t n, int mode,
    double histories, double voxel_volume_cm3, double calibration, float* dose, float* variance, uint32_t* counts_out,
    const JobCounters* counters, JobCounters* counters_out, cudaStream_t stream)
{
    const int block = 256;
    const int grid = static_cast<int>(std::min<uint64_t>((n + block - 1) / block, 152ull * 16));
    postprocess_records_kernel<float><<<grid, block, 0, stream>>>(records, w.palette_index ? nullptr : w.voxels, w.palette_index,
        w.palette, n, mode, histories, voxel_volume_cm3, calibration, dose, variance, counts_out, counters, counters_out);
    return cudaGetLastError();
}

cudaError_t launch_postprocess_f32(const float* tally, const WorldParams& w, uint64_t n, int mode, double histories,
    double voxel_volume_cm3, double calibration, double* dose, double* variance, const uint32_t* counts, uint32_t* counts_out,
    cudaStream_t stream)
{
    const int block = 256;
    const int grid = static_cast<int>(std::min<uint64_t>((n + block - 1) / block, 152ull * 16));
    postprocess_kernel<float><<<grid, block, 0, stream>>>(tally, w.palette_index ? nullptr : w.voxels, w.palette_index, w.palette, n, mode,
        histories, voxel_volume_cm3, calibration, dose, variance, counts, counts_out);
    return cudaGetLastError();
}

cudaError_t launch_max_density(const Voxel* voxels, uint64_t n, unsigned int* out_bits, int n_materials, cudaStream_t stream)
{
    const int block = 256;
    const int grid = static_cast<int>(std::min<uint64_t>((n + block - 1) / block, 152ull * 8));
    max_density_kernel<<<grid, block, n_materials * sizeof(unsigned int), stream>>>(voxels, n, out_bits, n_materials);
    return cudaGetLastError();
}

cudaError_t launch_probe_lut(const float* lut, LutMeta meta, int material, const double* energies, int n, double* out_att, double* out_maxinv, cudaStream_t stream)
{
    probe_lut_kernel<<<(n + 127) / 128, 128, 0, stream>>>(lut, meta, material, energies, n, out_att, out_maxinv);
    return cudaGetLastError();
}

cudaError_t launch_probe_interactions(const float* lut, LutMeta meta, int material, int model, int kind, float energy,
    uint64_t n, uint64_t seed, float* out_cos, float* out_energy, float* out_dep, cudaStream_t stream)
{
    const int block = 256;
    const int grid = static_cast<int>(std::min<uint64_t>((n + block - 1) / block, 152ull * 8));
    if (model == 0)
        probe_interactions_kernel<0><<<grid, block, 0, stream>>>(lut, meta, material, kind, energy, n, seed, out_cos, out_energy, out_dep);
    else if (model == 1)
        probe_interactions_kernel<1><<<grid, block, 0, stream>>>(lut, meta, material, kind, energy, n, seed, out_cos, out_energy, out_dep);
    else
        probe_interactions_kernel<2><<<grid, block, 0, stream>>>(lut, meta, material, kind, energy, n, seed, out_cos, out_energy, out_dep);
    return cudaGetLastError();
}

cudaError_t launch_probe_uniform(uint64_t seed, uint64_t n_streams, uint32_t draws, int kind, int nbins,
    unsigned long long* hist, int sm_count, cudaStream_t stream)
{
    const int block = 256;
    const int grid = static_cast<int>(std::min<uint64_t>((n_streams + block - 1) / block, static_cast<uint64_t>(sm_count) * 8));
    probe_uniform_kernel<<<grid, block, (nbins + 1) * sizeof(unsigned int), stream>>>(seed, n_streams, draws, kind, nbins, hist);
    return cudaGetLastError();
}

} // namespace dxmc_gb300::dev
