"""The single-job transport kernels on both sides of the shared-memory limit of the usual
one (tests/test_gpu_transport_variants.py has the other options): the job as it is routed
and the same job with a photon queue, which always runs the general kernel."""
from __future__ import annotations

import numpy as np
import pytest
from test_gpu_transport_variants import _run, _same, _source, _world

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", [0, 1, 2])
@pytest.mark.parametrize("materials,measured,energy", [(5, False, 150.0), (6, False, 150.0), (7, False, 150.0), (8, False, 80.0),
                                                       (6, True, 150.0), (8, True, 150.0)])
def test_jobs_around_the_shared_memory_limit(gpu_ctx, model, materials, measured, energy):
    import dxmclib_gb300 as dx
    w = _world(materials, measured, np.random.default_rng(materials))
    dworld = dx.DeviceWorld(gpu_ctx, w)
    dlut = dx.DeviceLut(gpu_ctx, dx.LutBlob(w.materialMap(), dworld.max_density(), energy))
    src = _source(60_001)
    _same(_run(gpu_ctx, dworld, dlut, src, model), _run(gpu_ctx, dworld, dlut, src, model, {"queue_log2_chunk": 17}))
    dlut.close()
    dworld.close()
