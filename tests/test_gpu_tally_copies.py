"""GPU tests of the copies of a pencil job's tally where memory is short: they only make
the job faster, so a budget that admits one copy admits the job, and copies that were
taken give way to whatever else needs the memory.  Results are those of a context with room:
counts equal, FP64 tallies to the order of their additions (relative 1e-9)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 96
RECORDS = N ** 3 * 32  # one copy of the tally
SLACK = 4 << 20        # tables, counters; far below a copy
HISTORIES = 1_000_000  # above the voxels: four copies where there is room


def _sources():
    import dxmclib_gb300 as dx
    from dxmclib_gb300.workloads import dx_source, pencil_water
    wl = pencil_water(n=N, histories=HISTORIES)
    field = dx_source(np.random.default_rng(5), 8, kvp=80.0)
    field.setTotalExposures(1)
    field.setHistoriesPerExposure(HISTORIES)
    return wl.world, wl.source, field


def _prepare(ctx, world):
    import dxmclib_gb300 as dx
    dworld = dx.DeviceWorld(ctx, world)
    dlut = dx.DeviceLut(ctx, dx.LutBlob(world.materialMap(), dworld.max_density(), 100.0))
    dworld.prepare(dlut)
    return dworld, dlut


@pytest.fixture(scope="module")
def expected(gpu_ctx):
    """Results with room, the bytes of what is resident beside jobs, and the memory of the pencil job."""
    import dxmclib_gb300 as dx
    from dxmclib_gb300 import _capi as A
    world, pencil, field = _sources()
    before = gpu_ctx.memory()[1]
    dworld, dlut = _prepare(gpu_ctx, world)
    resident = gpu_ctx.memory()[1] - before
    out, taken = [], []
    for src in (pencil, field):
        job = dx.Job(gpu_ctx, dworld, dlut, src.exposures(), getattr(src, "spectrum", lambda: None)(), None, None, seed=11, model=1)
        taken.append(gpu_ctx.memory()[1] - before - resident)
        out.append(job.result(A.OUTPUT_RAW))
        job.close()
    dlut.close()
    dworld.close()
    assert taken[0] > 4 * RECORDS and RECORDS < taken[1] < 2 * RECORDS
    return resident, out[0], out[1]


def _same(a, b):
    np.testing.assert_array_equal(a[2], b[2])
    for key in ("histories", "steps", "deposits"):
        assert a[3][key] == b[3][key]
    np.testing.assert_allclose(a[0], b[0], rtol=1e-9)
    np.testing.assert_allclose(a[1], b[1], rtol=1e-9)


def _pencil(ctx, dworld, dlut, src):
    import dxmclib_gb300 as dx
    return dx.Job(ctx, dworld, dlut, src.exposures(), None, None, None, seed=11, model=1)


def _field(ctx, dworld, dlut, src):
    import dxmclib_gb300 as dx
    return dx.Job(ctx, dworld, dlut, src.exposures(), src.spectrum(), None, None, seed=11, model=1)


def test_pencil_job_runs_where_one_copy_fits(expected):
    import dxmclib_gb300 as dx
    from dxmclib_gb300 import _capi as A
    resident, pencil_result, _ = expected
    world, pencil, _ = _sources()
    ctx = dx.GpuContext(memory_budget=resident + RECORDS + SLACK)
    dworld, dlut = _prepare(ctx, world)
    job = _pencil(ctx, dworld, dlut, pencil)
    _same(job.result(A.OUTPUT_RAW), pencil_result)
    job.close()
    ctx.close()


def test_copies_give_way_to_a_later_job(expected):
    """Room for the four copies of the first job, or for both jobs with one each: the second
    is admitted while the first runs, and the first keeps its result."""
    import dxmclib_gb300 as dx
    from dxmclib_gb300 import _capi as A
    resident, pencil_result, field_result = expected
    world, pencil, field = _sources()
    ctx = dx.GpuContext(memory_budget=resident + 4 * RECORDS + SLACK)
    dworld, dlut = _prepare(ctx, world)
    first = _pencil(ctx, dworld, dlut, pencil)
    assert ctx.memory()[1] > resident + 4 * RECORDS
    second = _field(ctx, dworld, dlut, field)
    assert ctx.memory()[1] < resident + 3 * RECORDS
    _same(second.result(A.OUTPUT_RAW), field_result)
    _same(first.result(A.OUTPUT_RAW), pencil_result)
    np.testing.assert_array_equal(first.preview(), first.result(A.OUTPUT_RAW)[0])
    first.close()
    second.close()
    assert ctx.memory()[1] == resident
    ctx.close()


def test_copies_give_way_within_a_batch(expected):
    import dxmclib_gb300 as dx
    from dxmclib_gb300 import _capi as A
    resident, pencil_result, field_result = expected
    world, pencil, field = _sources()
    ctx = dx.GpuContext(memory_budget=resident + 4 * RECORDS + SLACK)
    dworld, dlut = _prepare(ctx, world)
    batch = dx.Batch(ctx, [dx.BatchEntry(dworld, dlut, pencil.exposures(), seed=11, model=1),
                           dx.BatchEntry(dworld, dlut, field.exposures(), field.spectrum(), seed=11, model=1)])
    _same(batch.jobs[0].result(A.OUTPUT_RAW), pencil_result)
    _same(batch.jobs[1].result(A.OUTPUT_RAW), field_result)
    batch.close()
    assert ctx.memory()[1] == resident
    ctx.close()
