"""GPU test of how the persistent kernel's blocks share a batch: fewer jobs than the
block-wide search looks at together (32), just as many, one more and several rounds of
it; jobs of one history, around one chunk and of several chunks; chunks of 32 up.
Against the same jobs alone: histories, steps, deposits and event counts equal, tallies
up to the order of their additions (1e-9, as in test_gpu_batch.py)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = (1, 127, 128, 129, 33, 2000, 31, 256)


@pytest.mark.parametrize("n_jobs,chunk", [(1, 0), (31, 32), (32, 0), (33, 100), (97, 0)])
def test_blocks_share_jobs(gpu_ctx, n_jobs, chunk):
    import dxmclib_gb300 as dx
    world = dx.World()
    n = 12
    world.setDimensions((n, n, n))
    world.setSpacing((5.0, 5.0, 5.0))
    world.setDensityArray(np.ones(n ** 3))
    world.setMaterialIndexArray(np.zeros(n ** 3, np.uint8))
    world.addMaterialToMap(dx.Material("Water, Liquid"))
    src = dx.DXSource()
    src.setTotalExposures(1)
    src.setFieldSize((60.0, 60.0))
    src.updateFromWorld(world)
    src.validate()
    dworlds = [dx.DeviceWorld(gpu_ctx, world, layout=layout) for layout in (0, 1)]
    blob = dx.LutBlob(world.materialMap(), dworlds[0].max_density(), src.maxPhotonEnergyProduced())
    dlut = dx.DeviceLut(gpu_ctx, blob)
    args = []
    for k in range(n_jobs):
        src.setHistoriesPerExposure(SIZES[k % len(SIZES)])
        args.append((dworlds[k % 2], dlut, src.exposures(world.directionCosines()), src.spectrum(), src.heel(), src.bowtie(),
                     50 + k, k % 3))
    alone = [dx.Job(gpu_ctx, *a).result() for a in args]
    batch = dx.Batch(gpu_ctx, [dx.BatchEntry(*a) for a in args], mode=dx.Batch.PERSISTENT, item_histories=chunk)
    for k, (job, one) in enumerate(zip(batch.jobs, alone)):
        e, ee, counts, stats = job.result()
        assert stats["histories"] == one[3]["histories"] == SIZES[k % len(SIZES)]
        assert stats["steps"] == one[3]["steps"] and stats["deposits"] == one[3]["deposits"]
        np.testing.assert_array_equal(counts, one[2])
        np.testing.assert_allclose(e, one[0], rtol=1e-9, atol=0)
        np.testing.assert_allclose(ee, one[1], rtol=1e-9, atol=0)
    batch.close()
    dlut.close()
    for d in dworlds:
        d.close()
