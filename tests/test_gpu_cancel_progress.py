"""GPU tests of cancelling small jobs and of their progress: a job cancelled while it waits
behind another one takes no history, whichever kernel it would have run, a job of a few
rounds per warp stops while it runs, and its progress is in histories."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def body(gpu_ctx):
    import dxmclib_gb300 as dx
    from dxmclib_gb300.workloads import ct_helical
    wl = ct_helical(nz=64, histories=1_000_000)
    dworld = dx.DeviceWorld(gpu_ctx, wl.world)
    dlut = dx.DeviceLut(gpu_ctx, dx.LutBlob(wl.world.materialMap(), dworld.max_density(), wl.source.maxPhotonEnergyProduced()))
    yield wl.world, dworld, dlut
    dlut.close()
    dworld.close()


def _job(ctx, body, histories, launch=None, **kw):
    import dxmclib_gb300 as dx
    from dxmclib_gb300.workloads import ct_source
    world, dworld, dlut = body
    src = ct_source(world, histories)
    ex = src.exposures(world.directionCosines())
    job = dx.Job(ctx, dworld, dlut, ex, src.spectrum(), src.heel(), None, seed=3, model=1, launch=launch, **kw)
    return job, int(np.sum(ex.n_histories))


def _slow_job(ctx, body):
    """At most 24 rounds of 32 histories for each of its 608 warps, and tens of milliseconds."""
    from dxmclib_gb300 import _capi as A
    return _job(ctx, body, 400_000, launch=dict(blocks_per_sm=1, block_size=128), precision=A.PRECISION_FP64, tracking=A.TRACKING_GLOBAL)


@pytest.mark.parametrize("kind", ["usual", "global majorant", "FP64", "float tally"])
def test_job_cancelled_while_it_waits_takes_no_history(gpu_ctx, body, kind):
    from dxmclib_gb300 import _capi as A
    options = {"usual": {}, "global majorant": dict(tracking=A.TRACKING_GLOBAL), "FP64": dict(precision=A.PRECISION_FP64),
               "float tally": dict(tally_mode=A.TALLY_F32)}[kind]
    first, _ = _job(gpu_ctx, body, 1_000_000_000)
    job, total = _job(gpu_ctx, body, 1_000_000, **options)
    assert total > 900_000
    job.cancel()
    assert first.wait(0) == A.DXMC_ERR_TIMEOUT, "the first job was too short for this test"
    first.cancel()
    dose, var, nev, stats = job.result(A.OUTPUT_EV_PER_HISTORY, check=False)
    assert stats["status"] == A.DXMC_ERR_CANCELLED and stats["histories"] == 0
    assert not dose.any() and not var.any() and not nev.any()
    job.close()
    first.close()


def test_job_of_a_few_rounds_stops_while_it_runs(gpu_ctx, body):
    from dxmclib_gb300 import _capi as A
    job, total = _slow_job(gpu_ctx, body)
    while job.wait(0) == A.DXMC_ERR_TIMEOUT and job.progress()[0] == 0:
        pass
    assert job.wait(0) == A.DXMC_ERR_TIMEOUT, "the job was too short for this test"
    job.cancel()
    _, _, _, stats = job.result(A.OUTPUT_EV_PER_HISTORY, check=False)
    assert stats["status"] == A.DXMC_ERR_CANCELLED
    assert 0 < stats["histories"] < total
    job.close()


def test_progress_of_a_job_of_a_few_rounds(gpu_ctx, body):
    """The warps take their first units, about three quarters of such a job, when its kernel
    starts; then the progress grows with the small units that are taken."""
    from dxmclib_gb300 import _capi as A
    job, total = _slow_job(gpu_ctx, body)
    seen = []
    while True:
        started, of = job.progress()
        if job.wait(0) != A.DXMC_ERR_TIMEOUT:
            break
        assert of == total
        if started:
            seen.append(started)
    assert len(seen) > 2, "the job was too short for this test"
    assert seen == sorted(seen) and seen[-1] <= total
    assert total // 2 < seen[0] < total
    assert job.progress() == (total, total)
    job.close()
