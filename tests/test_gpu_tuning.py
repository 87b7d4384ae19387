"""Every number of blocks per SM the tuning accepts gives the same lists, and the
largest is not slower than the default (4)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_blocks_per_sm():
    import gpuequiv_b200 as geq
    from gpuequiv_b200 import synth
    ctx = geq.Context(0)
    g = geq.GameGraph.from_csr(*synth.scaled_stress_game(2, 1_500_000, 6_000_000), geq.EnergyConf.STANDARD)
    dg = geq.DeviceGames([g], ctx)
    ms, lists = {}, {}
    for bps in (4, 5, 2, 3, 4, 5):
        ctx.set_tuning(blocks_per_sm=bps)
        dg.solve()
        ms[bps] = min([ms.get(bps, 1e9)] + [dg.solve()["device_ms"] for _ in range(7)])
        offs, data, _ = geq.run_batch_raw([g], ctx)
        o = offs[0].astype(np.int64)
        # lists are sets: sorted within a position
        lists[bps] = (o, data[0][np.lexsort((data[0], np.repeat(np.arange(len(o) - 1), np.diff(o))))])
    for bps in (2, 3, 5):
        assert all(np.array_equal(a, b) for a, b in zip(lists[bps], lists[4]))
    assert ms[5] < 1.06 * ms[4], ms
    ctx.close()
