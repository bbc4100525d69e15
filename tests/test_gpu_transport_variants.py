"""The single-job transport kernels against each other: the kernel of the usual options
and the general one (a job with a pre-generated photon queue runs it) follow the same
histories, so counts and counters are equal and the FP64 tallies differ by the order of
their additions only (relative 1e-9).  Material counts at the edge of the attenuation
table, with and without a measurement map, both voxel layouts, all models, and history
counts at the edges of the work split (fewer than a warp, one unit short of and past a
round of the device, several rounds)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAMES = ("Water, Liquid", "Bone, Cortical (ICRP)", "Air, Dry (near sea level)", "Tissue, Soft (ICRP)", "Lung Tissue (ICRU-44)")


def _world(materials, measured, rng):
    import dxmclib_gb300 as dx
    dims = (21, 17, 19)
    n = int(np.prod(dims))
    mat = rng.integers(0, materials, n).astype(np.uint8)
    w = dx.World()
    w.setDimensions(dims)
    w.setSpacing((5.0, 6.0, 4.0))
    w.setDensityArray((0.6 + 0.4 * (mat % 3)).astype(np.float32))
    w.setMaterialIndexArray(mat)
    if measured:
        w.setMeasurementMapArray((rng.random(n) < 0.05).astype(np.uint8))
    for k in range(materials):
        w.addMaterialToMap(dx.Material(NAMES[k % len(NAMES)]))
    assert w.isValid()
    return w


def _run(ctx, dworld, dlut, src, model, launch=None):
    import dxmclib_gb300 as dx
    from dxmclib_gb300 import _capi as A
    job = dx.Job(ctx, dworld, dlut, src.exposures(), src.spectrum(), src.heel(), None, seed=11, model=model, launch=launch)
    out = job.result(A.OUTPUT_RAW)
    job.close()
    return out


def _same(a, b):
    np.testing.assert_array_equal(a[2], b[2])
    for key in ("histories", "steps", "deposits"):
        assert a[3][key] == b[3][key]
    assert a[3]["rejection_overflows"] == b[3]["rejection_overflows"] == 0
    np.testing.assert_allclose(a[0], b[0], rtol=1e-9)
    np.testing.assert_allclose(a[1], b[1], rtol=1e-9)


def _source(histories):
    from dxmclib_gb300.workloads import dx_source
    src = dx_source(np.random.default_rng(5), 8, kvp=80.0)
    src.setTotalExposures(1)
    src.setHistoriesPerExposure(histories)
    return src


@pytest.mark.parametrize("model", [0, 1, 2])
@pytest.mark.parametrize("materials,measured,layout", [(1, False, 0), (8, False, 0), (9, False, 0), (8, True, 0), (9, True, 1), (8, False, 1)])
def test_usual_and_general_kernels_agree(gpu_ctx, model, materials, measured, layout):
    import dxmclib_gb300 as dx
    w = _world(materials, measured, np.random.default_rng(materials))
    dworld = dx.DeviceWorld(gpu_ctx, w, layout=layout)
    dlut = dx.DeviceLut(gpu_ctx, dx.LutBlob(w.materialMap(), dworld.max_density(), 150.0))
    src = _source(60_001)
    _same(_run(gpu_ctx, dworld, dlut, src, model), _run(gpu_ctx, dworld, dlut, src, model, {"queue_log2_chunk": 17}))
    dlut.close()
    dworld.close()


@pytest.mark.parametrize("histories", [1, 31, 33, 155_647, 155_649, 311_297, 500_003, 4_000_037])
def test_work_split_takes_every_history_once(gpu_ctx, histories):
    """155 648 histories are one round of 32 for 152 SMs of four eight-warp blocks (of
    nine warps: 175 104)."""
    import dxmclib_gb300 as dx
    w = _world(2, False, np.random.default_rng(2))
    dworld = dx.DeviceWorld(gpu_ctx, w)
    dlut = dx.DeviceLut(gpu_ctx, dx.LutBlob(w.materialMap(), dworld.max_density(), 150.0))
    src = _source(histories)
    usual = _run(gpu_ctx, dworld, dlut, src, 1)
    assert usual[3]["histories"] == histories
    _same(usual, _run(gpu_ctx, dworld, dlut, src, 1, {"queue_log2_chunk": 19}))
    dlut.close()
    dworld.close()


@pytest.mark.parametrize("model", [1, 2])
@pytest.mark.parametrize("histories", [499_990, 500_000, 700_010])
def test_pencil_tally_copies(gpu_ctx, model, histories):
    """A pencil beam's job of 5e5 histories or more adds to copies of the tally; a member
    of a persistent batch has one.  A finished job's preview is its raw energy tally."""
    import dxmclib_gb300 as dx
    from dxmclib_gb300 import _capi as A
    w = _world(2, False, np.random.default_rng(3))
    dworld = dx.DeviceWorld(gpu_ctx, w)
    dlut = dx.DeviceLut(gpu_ctx, dx.LutBlob(w.materialMap(), dworld.max_density(), 150.0))
    src = dx.PencilSource()
    src.setPosition((0.0, 0.0, -200.0))
    src.setDirectionCosines((1, 0, 0, 0, 1, 0))
    src.setPhotonEnergy(60.0)
    src.setTotalExposures(10)
    src.setHistoriesPerExposure(histories // 10)
    job = dx.Job(gpu_ctx, dworld, dlut, src.exposures(), seed=11, model=model)
    alone = job.result(A.OUTPUT_RAW)
    np.testing.assert_array_equal(job.preview(), alone[0])
    job.close()
    batch = dx.Batch(gpu_ctx, [dx.BatchEntry(dworld, dlut, src.exposures(), seed=11, model=model)], mode=dx.Batch.PERSISTENT)
    _same(alone, batch.jobs[0].result(A.OUTPUT_RAW))
    batch.close()
    dlut.close()
    dworld.close()
