// Siddon traversal: the radiological path of straight rays through the voxel
// grid.  DXMClib has no counterpart (it tracks photons with Woodcock steps only);
// the kernel serves primary-transmission and projection computations on the
// same resident world and LUT as the transport.
//
// One thread per ray, incremental form (Jacobs et al., Int. J. Imaging Syst.
// Technol. 1998): after the slab intersection with the grid box, the ray moves
// from one voxel boundary plane to the next, taking the nearest of the three
// next crossings, and adds mu / rho x density x segment length.
//
// The kernel is bound by instruction issue: a warp's rays lie side by side, so
// their voxels come from L1, and what counts is the number of instructions per
// crossed voxel.  mu / rho is evaluated once per ray for every material (or mu
// for every palette entry) and kept in shared memory, one column per thread: on
// demand, some lane of a warp met a new material in most steps and the whole
// warp paid for three exponentials each time.  The three axes live in registers
// (no indexed arrays), a linear voxel offset and per-axis counts of the planes
// left replace the index triple, and a voxel is read one step before its length
// is added, so its latency hides behind the next plane.  Up to a distance at which
// no axis can have left the grid, whatever the rounding, the steps go without the
// counts and without the test for the ray's end: 31 instructions a step where there
// were 44; the last few steps of a ray and the first take the checked form.  2^20 rays
// through the 512 x 512 x 200 CT body: 4.54 ms with the attenuation on demand, 1.04 ms
// with the tables, 0.71 ms with the unchecked steps (121 k, 27.6 k and 19.2 k thread
// instructions per ray).  What is left is L1: eight lines a read, 92 % of the wavefronts
// that it can serve.
#include "transport.cuh"

namespace dxmc_gb300::dev {
namespace {

    // Where a segment's attenuation comes from: a per-ray table of mu per palette
    // entry, a per-ray table of mu / rho per material, or the LUT on demand.
    enum : int { BY_ENTRY = 0, BY_MATERIAL = 1, ON_DEMAND = 2 };
    // Columns of the per-ray table.  A column costs one evaluation per ray (about 40
    // instructions; a ray of the CT body takes 20 per voxel over hundreds of voxels)
    // and 512 bytes of shared memory per block, which at 8 still leaves every SM its
    // full count of resident warps.
    constexpr int MU_COLUMNS = 8;
    constexpr int PATH_THREADS = 128;

    // A voxel as read from the grid, and the integer that indexes the grid (compact
    // worlds hold fewer than 2^32 voxels).
    template <bool PALETTE>
    struct RawVoxel {
        uint2 v;
    };
    template <>
    struct RawVoxel<true> {
        uint32_t v;
    };
    template <bool PALETTE>
    struct VoxelIndex {
        using type = uint64_t;
    };
    template <>
    struct VoxelIndex<true> {
        using type = uint32_t;
    };

    template <bool PALETTE>
    __device__ __forceinline__ RawVoxel<PALETTE> read_voxel(const WorldParams& w, typename VoxelIndex<PALETTE>::type i)
    {
        if constexpr (PALETTE)
            return RawVoxel<true> { __ldg(w.palette_index + i) };
        else
            return RawVoxel<false> { __ldg(reinterpret_cast<const uint2*>(w.voxels) + i) };
    }

    struct MaterialVoxel {
        float density;
        int mat;
    };

    __device__ __forceinline__ MaterialVoxel entry_voxel(const PaletteEntry& e)
    {
        return MaterialVoxel { e.density, static_cast<int>(e.code & 0xffu) };
    }

    template <bool PALETTE, int MU>
    __global__ void __launch_bounds__(PATH_THREADS) radiological_path_kernel(const __grid_constant__ WorldParams w, const float* __restrict__ L,
        const __grid_constant__ LutMeta m, const float* __restrict__ rays, uint64_t n, double* __restrict__ out)
    {
        using Index = typename VoxelIndex<PALETTE>::type;
        __shared__ float table[MU == ON_DEMAND ? 1 : MU_COLUMNS][PATH_THREADS];
        const int tid = threadIdx.x;
        const auto mu_over_rho = [&](int mat, float logE, int seg) {
            float a0, a1, a2;
            lut_attenuation(L, m, mat, logE, seg, a0, a1, a2);
            return a0 + a1 + a2;
        };
        for (uint64_t r = blockIdx.x * static_cast<uint64_t>(blockDim.x) + tid; r < n; r += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
            const float* ray = rays + 7 * r;
            float o[3] = { ray[0], ray[1], ray[2] };
            float d[3] = { ray[3], ray[4], ray[5] };
            const float energy = ray[6];
            const float norm = sqrtf(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
            double result = 0.0;
            if (norm > 0.0f && energy > 0.0f) {
#pragma unroll
                for (int k = 0; k < 3; ++k)
                    d[k] /= norm;
                // slab intersection with the grid box, forward part of the ray only
                float tmin = 0.0f, tmax = INFINITY;
                bool hit = true;
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const float lo = w.lower[k];
                    const float hi = w.lower[k] + w.spacing[k] * static_cast<float>(w.dims[k]);
                    if (d[k] != 0.0f) {
                        const float t1 = (lo - o[k]) / d[k];
                        const float t2 = (hi - o[k]) / d[k];
                        tmin = fmaxf(tmin, fminf(t1, t2));
                        tmax = fminf(tmax, fmaxf(t1, t2));
                    } else if (o[k] < lo || o[k] >= hi) {
                        hit = false;
                    }
                }
                if (hit && tmax > tmin) {
                    // per axis: the next crossing, the spacing of the crossings, the voxels
                    // left in the direction of the ray and the change of the voxel offset
                    float tnext[3], dt[3];
                    int left[3];
                    Index move[3];
                    Index voxel = 0;
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const Index stride = k == 0 ? Index(1) : (k == 1 ? static_cast<Index>(w.dims[0]) : static_cast<Index>(w.nxy));
                        // voxel of the first segment's midpoint-side: entry point nudged along the ray
                        const float p = o[k] + d[k] * tmin;
                        int i = static_cast<int>(floorf((p - w.lower[k]) / w.spacing[k]));
                        if (d[k] < 0.0f && p - w.lower[k] == static_cast<float>(i) * w.spacing[k])
                            --i; // on a boundary plane moving down: the voxel below
                        i = min(max(i, 0), static_cast<int>(w.dims[k]) - 1);
                        voxel += static_cast<Index>(i) * stride;
                        if (d[k] > 0.0f) {
                            left[k] = static_cast<int>(w.dims[k]) - 1 - i;
                            move[k] = stride;
                            tnext[k] = (w.lower[k] + static_cast<float>(i + 1) * w.spacing[k] - o[k]) / d[k];
                            dt[k] = w.spacing[k] / d[k];
                        } else if (d[k] < 0.0f) {
                            left[k] = i;
                            move[k] = Index(0) - stride;
                            tnext[k] = (w.lower[k] + static_cast<float>(i) * w.spacing[k] - o[k]) / d[k];
                            dt[k] = -w.spacing[k] / d[k];
                        } else {
                            left[k] = 0;
                            move[k] = 0;
                            tnext[k] = INFINITY;
                            dt[k] = INFINITY;
                        }
                    }
                    const float logE = log10f(energy);
                    const int seg = lut_segment(L, m, logE);
                    if constexpr (MU == BY_ENTRY) {
                        for (int e = 0; e < w.palette_n; ++e) {
                            const MaterialVoxel v = entry_voxel(w.palette[e]);
                            table[e][tid] = mu_over_rho(v.mat, logE, seg) * v.density;
                        }
                    } else if constexpr (MU == BY_MATERIAL) {
                        for (int mat = 0; mat < m.n_materials; ++mat)
                            table[mat][tid] = mu_over_rho(mat, logE, seg);
                    }
                    int cached = -1;
                    float mu_rho = 0.0f;
                    float t = tmin;
                    float acc = 0.0f, comp = 0.0f; // compensated sum of mu * length (mm)
                    float length = -1.0f;          // of the segment whose voxel has been read, not yet added (< 0: none)
                    RawVoxel<PALETTE> raw {};
                    const auto add = [&]() {
                        float mu;
                        if constexpr (MU == BY_ENTRY) {
                            mu = table[raw.v][tid];
                        } else {
                            MaterialVoxel v;
                            if constexpr (PALETTE)
                                v = entry_voxel(w.palette[raw.v]);
                            else
                                v = MaterialVoxel { __uint_as_float(raw.v.x), static_cast<int>(raw.v.y & 0xffu) };
                            if constexpr (MU == BY_MATERIAL) {
                                mu = table[v.mat][tid] * v.density;
                            } else {
                                if (v.mat != cached) {
                                    mu_rho = mu_over_rho(v.mat, logE, seg);
                                    cached = v.mat;
                                }
                                mu = mu_rho * v.density;
                            }
                        }
                        const float y = fmaf(mu, length, -comp);
                        const float s = acc + y;
                        comp = (s - acc) - y;
                        acc = s;
                    };
                    // No axis can leave the grid before t_safe: the crossing that leaves it by
                    // axis k is the one after left[k] more, at tnext + left dt in exact
                    // arithmetic, and each of the additions that lead there rounds by at most
                    // 2^-24 of the largest term.  Twice that is taken off.
                    float t_safe = tmax;
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        if (d[k] != 0.0f) {
                            const float leaves = left[k] ? fmaf(static_cast<float>(left[k]), dt[k], tnext[k]) : tnext[k];
                            const float slack = static_cast<float>(left[k] + 4) * 0x1p-23f * fmaxf(fabsf(leaves), fabsf(tnext[k]));
                            t_safe = leaves - slack < INFINITY ? fminf(t_safe, leaves - slack) : -INFINITY;
                        }
                    }
                    // ends at the last voxel of an axis (left < 0): at most the sum of the dimensions
                    while (true) {
                        const bool x_first = tnext[0] <= tnext[1];
                        const float txy = x_first ? tnext[0] : tnext[1];
                        const bool xy_first = txy <= tnext[2];
                        const float tk = xy_first ? txy : tnext[2];
                        const float tn = fminf(tk, tmax);
                        if (tn > t) {
                            if (length >= 0.0f)
                                add();
                            raw = read_voxel<PALETTE>(w, voxel);
                            length = tn - t;
                            t = tn;
                        }
                        if (tk >= tmax)
                            break;
                        if (xy_first && x_first) {
                            voxel += move[0];
                            --left[0];
                            tnext[0] += dt[0];
                        } else if (xy_first) {
                            voxel += move[1];
                            --left[1];
                            tnext[1] += dt[1];
                        } else {
                            voxel += move[2];
                            --left[2];
                            tnext[2] += dt[2];
                        }
                        if ((left[0] | left[1] | left[2]) < 0)
                            break;
                        if (length < 0.0f || !(t_safe > 0.0f))
                            continue;
                        // the same steps up to t_safe, without the counts and the end of the ray
                        while (true) {
                            const float tk = fminf(fminf(tnext[0], tnext[1]), tnext[2]);
                            if (!(tk < t_safe))
                                break;
                            const bool step_x = tnext[0] == tk;
                            const bool step_y = !step_x && tnext[1] == tk;
                            const bool step_z = !step_x && !step_y;
                            if (tk > t) {
                                add();
                                raw = read_voxel<PALETTE>(w, voxel);
                                length = tk - t;
                                t = tk;
                            }
                            if (step_x) {
                                voxel += move[0];
                                tnext[0] += dt[0];
                            }
                            if (step_y) {
                                voxel += move[1];
                                tnext[1] += dt[1];
                            }
                            if (step_z) {
                                voxel += move[2];
                                tnext[2] += dt[2];
                            }
                        }
                        t_safe = -INFINITY;
                        const Index nx = static_cast<Index>(w.dims[0]), nxy = static_cast<Index>(w.nxy);
                        const int at[3] = { static_cast<int>(voxel % nx), static_cast<int>(voxel % nxy / nx), static_cast<int>(voxel / nxy) };
#pragma unroll
                        for (int k = 0; k < 3; ++k)
                            left[k] = d[k] > 0.0f ? static_cast<int>(w.dims[k]) - 1 - at[k] : (d[k] < 0.0f ? at[k] : 0);
                    }
                    if (length >= 0.0f)
                        add();
                    result = 0.1 * static_cast<double>(acc); // mm -> cm
                }
            }
            out[r] = result;
        }
    }

    template <bool PALETTE, int MU>
    void launch_path(const WorldParams& w, const float* lut, const LutMeta& meta, const float* rays, uint64_t n, double* out, cudaStream_t stream)
    {
        // Blocks of a warp while those leave SMs without one, so that a few thousand rays
        // spread over the device.  Above that, blocks of 128 and one ray per thread: rays
        // differ in length, so smaller blocks free their SM earlier (256 threads in at most
        // 152 x 32 blocks: 0.03 ms more for 2^20 rays; blocks of 32 and 64 equal).
        int block = PATH_THREADS;
        while (block > 32 && (n + block - 1) / block < 2 * 152)
            block /= 2;
        const int grid = static_cast<int>(std::min<uint64_t>((n + block - 1) / block, 1u << 30));
        radiological_path_kernel<PALETTE, MU><<<grid, block, 0, stream>>>(w, lut, meta, rays, n, out);
    }

} // namespace

cudaError_t launch_radiological_path(const WorldParams& w, const float* lut, LutMeta meta, const float* rays, uint64_t n,
    double* out, cudaStream_t stream)
{
    const bool materials_fit = meta.n_materials <= MU_COLUMNS;
    if (w.palette_index) {
        if (w.palette_n <= MU_COLUMNS)
            launch_path<true, BY_ENTRY>(w, lut, meta, rays, n, out, stream);
        else if (materials_fit)
            launch_path<true, BY_MATERIAL>(w, lut, meta, rays, n, out, stream);
        else
            launch_path<true, ON_DEMAND>(w, lut, meta, rays, n, out, stream);
    } else if (materials_fit) {
        launch_path<false, BY_MATERIAL>(w, lut, meta, rays, n, out, stream);
    } else {
        launch_path<false, ON_DEMAND>(w, lut, meta, rays, n, out, stream);
    }
    return cudaGetLastError();
}

} // namespace dxmc_gb300::dev
