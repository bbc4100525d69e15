"""GPU test of the context's block size: sizes that are no whole warps run as whole warps,
and every size takes every history once."""
from __future__ import annotations

import numpy as np
import pytest
from test_gpu_transport_variants import _run, _same, _source, _world

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block_size", [1, 32, 98, 100, 256])
def test_every_block_size_takes_every_history_once(gpu_ctx, block_size):
    import dxmclib_gb300 as dx
    w = _world(2, False, np.random.default_rng(2))
    src = _source(200_003)
    results = []
    for ctx in (gpu_ctx, dx.GpuContext(block_size=block_size)):
        dworld = dx.DeviceWorld(ctx, w)
        dlut = dx.DeviceLut(ctx, dx.LutBlob(w.materialMap(), dworld.max_density(), 150.0))
        results.append(_run(ctx, dworld, dlut, src, 1))
        dlut.close()
        dworld.close()
        if ctx is not gpu_ctx:
            ctx.close()
    assert results[0][3]["histories"] == 200_003
    _same(results[1], results[0])
