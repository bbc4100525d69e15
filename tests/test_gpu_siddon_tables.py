"""GPU test of the Siddon kernel's attenuation tables: worlds whose palette entries
or materials just fit the per-ray table (8 columns) or just do not, for both voxel
layouts and ray counts at the edges of the kernel's block sizes, against the CPU
restatement in oracle/siddon.py.  Tolerance as in test_gpu_siddon.py (FP32 LUT,
compensated FP32 sum)."""
from __future__ import annotations

import sys
from pathlib import Path

import numpy as np
import pytest

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "oracle"))
import siddon  # noqa: E402
from test_gpu_siddon import _rays  # noqa: E402

pytestmark = pytest.mark.gpu

NAMES = ("Water, Liquid", "Bone, Cortical (ICRP)", "Air, Dry (near sea level)", "Tissue, Soft (ICRP)", "Lung Tissue (ICRU-44)")


@pytest.mark.parametrize("materials,densities,layout,n_rays", [
    (1, 1, 0, 1), (2, 4, 0, 31), (8, 1, 0, 33), (3, 3, 0, 257), (9, 1, 0, 129), (8, 2, 0, 1000), (8, 2, 1, 63), (9, 1, 1, 255)])
def test_path_tables_match_cpu(gpu_ctx, materials, densities, layout, n_rays):
    import dxmclib_gb300 as dx
    rng = np.random.default_rng(materials * 100 + densities * 10 + layout)
    dims, sp = (13, 9, 11), (2.0, 2.5, 3.0)
    n = int(np.prod(dims))
    mat = rng.integers(0, materials, n).astype(np.uint8)
    dens = (0.5 + 0.25 * rng.integers(0, densities, n)).astype(np.float32)
    world = dx.World()
    world.setDimensions(dims)
    world.setSpacing(sp)
    world.setDensityArray(dens)
    world.setMaterialIndexArray(mat)
    for k in range(materials):
        world.addMaterialToMap(dx.Material(NAMES[k % len(NAMES)]))
    assert world.isValid()
    dworld = dx.DeviceWorld(gpu_ctx, world, layout=layout)
    blob = dx.LutBlob(world.materialMap(), dworld.max_density(), 150.0)
    dlut = dx.DeviceLut(gpu_ctx, blob)
    ext = np.array(world.matrixExtent()).reshape(3, 2)
    lo, hi = ext[:, 0], ext[:, 1]
    rays = _rays(lo, hi, rng, max(n_rays, 4))[:n_rays]
    gpu = dworld.radiological_path(dlut, rays)
    cpu = siddon.radiological_path(dims, sp, lo, dens, mat, lambda m, e: float(np.sum(blob.attenuation(m, e))),
                                   rays.astype(np.float64))
    np.testing.assert_allclose(gpu, cpu, rtol=1e-4, atol=1e-6 * cpu.max())
    dlut.close()
    dworld.close()


@pytest.mark.parametrize("dims", [(1, 1, 1), (1, 40, 3), (70, 2, 5), (2, 3, 150), (33, 31, 32)])
@pytest.mark.parametrize("shift", [0.0, 700.0])
def test_path_ends_at_the_grid(gpu_ctx, dims, shift):
    """Thin, long and shifted grids, where the unchecked steps end close to where an
    axis runs out of voxels: rays along the axes, along diagonals and in general
    directions, from inside and from outside."""
    import dxmclib_gb300 as dx
    rng = np.random.default_rng(int(np.prod(dims)) + int(shift))
    sp = (2.0, 2.5, 3.0)
    n = int(np.prod(dims))
    mat = rng.integers(0, 3, n).astype(np.uint8)
    dens = (0.5 + 0.25 * rng.integers(0, 3, n)).astype(np.float32)
    world = dx.World()
    world.setDimensions(dims)
    world.setSpacing(sp)
    world.setOrigin((shift, -shift, 0.5 * shift))
    world.setDensityArray(dens)
    world.setMaterialIndexArray(mat)
    for name in NAMES[:3]:
        world.addMaterialToMap(dx.Material(name))
    assert world.isValid()
    dworld = dx.DeviceWorld(gpu_ctx, world)
    blob = dx.LutBlob(world.materialMap(), dworld.max_density(), 150.0)
    dlut = dx.DeviceLut(gpu_ctx, blob)
    ext = np.array(world.matrixExtent()).reshape(3, 2)
    lo = ext[:, 0]
    count = 600
    rays = np.zeros((count, 7), dtype=np.float32)
    inside = lo + (np.floor(rng.uniform(0, 1, (count, 3)) * dims) + rng.uniform(0.1, 0.9, (count, 3))) * sp
    direction = rng.normal(size=(count, 3))
    direction[:200] = np.eye(3)[rng.integers(0, 3, 200)] * rng.choice([-1.0, 1.0], (200, 1))
    direction[200:400] = np.asarray(sp) * rng.choice([-1.0, 1.0], (200, 3))
    direction /= np.linalg.norm(direction, axis=1, keepdims=True)
    rays[:, 3:6] = direction
    rays[:, :3] = inside - direction * rng.choice([0.0, 400.0], (count, 1))
    rays[:, 6] = rng.uniform(15, 140, count)
    gpu = dworld.radiological_path(dlut, rays)
    cpu = siddon.radiological_path(dims, sp, lo, dens, mat, lambda m, e: float(np.sum(blob.attenuation(m, e))),
                                   rays.astype(np.float64))
    # positions and distances of 1000 mm in FP32 move a crossing by 1e-4 mm over the
    # component of the direction, and a chord is 0.2 mm over it or longer: 5e-4 an end
    np.testing.assert_allclose(gpu, cpu, rtol=1e-4, atol=1e-3 * float(cpu.max()))
    dlut.close()
    dworld.close()
