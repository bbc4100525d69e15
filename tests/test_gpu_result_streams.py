"""GPU test of results beside running jobs: the large pageable result of a job that has ended
does not wait for a running job whose asynchronous result is pending.  (The running job
leaves room on the SMs: the results' kernel would wait for one that fills them.)"""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_pageable_result_does_not_wait_for_another_job(gpu_ctx):
    import dxmclib_gb300 as dx
    from dxmclib_gb300 import _capi as A
    from dxmclib_gb300.workloads import ct_helical, ct_source
    wl = ct_helical(nz=64, histories=2_000_000)  # 16.8 M voxels: 336 MB of results

    def job(src, launch=None):
        return dx.Job(gpu_ctx, dworld, dlut, src.exposures(wl.world.directionCosines()), src.spectrum(), src.heel(), None, seed=3, model=1, launch=launch)

    dworld = dx.DeviceWorld(gpu_ctx, wl.world)
    dlut = dx.DeviceLut(gpu_ctx, dx.LutBlob(wl.world.materialMap(), dworld.max_density(), wl.source.maxPhotonEnergyProduced()))
    first = job(wl.source)
    assert first.wait() == A.DXMC_OK
    expected = first.result(A.OUTPUT_RAW)
    running = job(ct_source(wl.world, 1_000_000_000), dict(blocks_per_sm=1, block_size=128))
    pinned = torch.zeros(wl.world.size(), dtype=torch.float64, pin_memory=True).numpy()
    running.result_async(A.OUTPUT_RAW, out=(pinned, None, None))
    again = first.result(A.OUTPUT_RAW)
    assert running.wait(0) == A.DXMC_ERR_TIMEOUT
    for a, b in zip(again[:3], expected[:3]):
        np.testing.assert_array_equal(a, b)
    running.cancel()
    running.result_wait(check=False)
    for obj in (running, first, dlut, dworld):
        obj.close()
