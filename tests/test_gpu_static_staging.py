"""Lone games are copied by the solving kernel itself from a staging block that
earlier calls used: what those left in front of the game (where the device block
has its control block) must not reach it."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from helpers import canon
from oracle import ora

pytestmark = pytest.mark.gpu


def game(n, seed):
    rng = np.random.default_rng(seed)
    att = (rng.random(n) < 0.6).astype(np.uint8)
    deg = rng.integers(0, 4, n)
    row = np.zeros(n + 1, np.uint32)
    np.cumsum(deg, out=row[1:])
    m = int(row[-1])
    col = rng.integers(0, n, m).astype(np.uint32)
    wt = np.where(rng.random(m) < 0.5, np.uint32(1) << (4 * rng.integers(0, 6, m)).astype(np.uint32), 0)
    return row, col, wt.astype(np.uint32), att


@pytest.mark.parametrize("n", [1, 80, 257, 401, 5000])
def test_dirty_staging(n):
    import gpuequiv_b200 as geq
    from gpuequiv_b200._lib import check, geq_energy_lists, lib
    ctx = geq.Context(0)
    # two games at once are packed from the staging block's first byte on:
    # row offsets of 16,000 one-edge positions fill it with large words
    big = 16000
    filler = geq.GameGraph.from_csr(np.arange(big + 1, dtype=np.uint32), np.full(big, big - 1, np.uint32),
                                    np.zeros(big, np.uint32), np.ones(big, np.uint8), geq.EnergyConf.STANDARD)
    g = game(n, n)
    small = geq.GameGraph.from_csr(*g, geq.EnergyConf.STANDARD)
    reach = np.nonzero((g[3] == 0) & (np.diff(g[0].astype(np.int64)) == 0))[0].astype(np.uint32)
    exp = ora.run_game(6, 3, *g, reach).lists()
    for _ in range(3):
        for graphs in ([filler, filler], [small]):
            views = geq.c_views(graphs)
            sol, out = C.c_void_p(), geq_energy_lists()
            check(lib.geq_energy_game_run_batch(ctx.h, len(graphs), views, None, None, None, C.byref(sol)))
            check(lib.geq_solution_lists(sol, 0, C.byref(out)))
            if len(graphs) == 1:
                o = np.ctypeslib.as_array(out.offsets, shape=(n + 1,)).astype(np.int64)
                d = np.ctypeslib.as_array(out.data, shape=(int(o[-1]),)).copy() if o[-1] else np.zeros(0, np.uint32)
                for v in range(n):
                    assert canon(d[o[v]:o[v + 1]]) == canon(exp[v]), f"position {v}"
            lib.geq_solution_free(sol)
    ctx.close()
