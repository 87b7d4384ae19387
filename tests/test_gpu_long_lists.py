"""Lists on their way to the host: short ones by a thread each, ones of more
than 16 energies by a warp, a warp per position where all are long -- in whole
downloads, in the server's and in a lone game's launch."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from oracle import ora

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def geq():
    import gpuequiv_b200 as geq
    return geq


@pytest.fixture(scope="module")
def ctx(geq):
    c = geq.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 3000])
@pytest.mark.parametrize("lengths", [(0, 1, 5, 6), (15, 16, 17), (16,), (17,), (1, 2, 1, 0, 500), (33, 300, 580)])
def test_given_lists(geq, ctx, n, lengths):
    """Positions without successors keep the lists they were given, in order."""
    from gpuequiv_b200._lib import check, geq_energy_lists, lib
    rng = np.random.default_rng(n)
    e = np.array(np.meshgrid(*[np.arange(4)] * 6)).reshape(6, -1).T
    words = (e[e.sum(1) == 9] << (2 * np.arange(6))).sum(1).astype(np.uint32)  # 580, none below another
    counts = np.array(lengths)[rng.integers(0, len(lengths), n)]
    offs = np.zeros(n + 1, np.uint64)
    offs[1:] = np.cumsum(counts)
    data = np.concatenate([rng.permutation(words)[:k] for k in counts] + [words[:1]]).astype(np.uint32)
    g = geq.GameGraph.from_csr(np.zeros(n + 1, np.uint32), np.zeros(0, np.uint32), np.zeros(0, np.uint32),
                               np.ones(n, np.uint8), geq.EnergyConf.STANDARD)
    view = g.c_view()
    init = geq_energy_lists(n, 1, offs.ctypes.data_as(C.POINTER(C.c_uint64)),
                            data.ctypes.data_as(C.POINTER(C.c_uint32)))
    sol, out = C.c_void_p(), geq_energy_lists()
    check(lib.geq_energy_game_run(ctx.h, C.byref(view), C.byref(init), None, 0, C.byref(sol)))
    check(lib.geq_solution_lists(sol, 0, C.byref(out)))
    o = np.ctypeslib.as_array(out.offsets, shape=(n + 1,)).copy()
    d = np.ctypeslib.as_array(out.data, shape=(int(o[-1]),)).copy() if o[-1] else np.zeros(0, np.uint32)
    lib.geq_solution_free(sol)
    assert np.array_equal(o, offs)
    assert np.array_equal(d, data[:int(offs[-1])])


@pytest.mark.parametrize("width", [1, 40, 300])
def test_grown_lists(geq, ctx, width):
    """Layers of positions with 1, 6, 21, 56, 96, ... energies, alone (one
    block, a cluster), beside an empty game and through the server."""
    from gpuequiv_b200.serving import Server
    depth = 6
    row = np.concatenate([np.zeros(width), np.arange(width * depth + 1) * 6]).astype(np.uint32)
    rng = np.random.default_rng(width)
    col = (np.repeat(np.arange(depth) * width, width * 6) + rng.integers(0, width, width * depth * 6)).astype(np.uint32)
    wt = np.tile(np.uint32(1) << (4 * np.arange(6)).astype(np.uint32), width * depth).astype(np.uint32)
    att = (np.arange(width * (depth + 1)) >= width).astype(np.uint8)
    exp = [np.sort(np.asarray(x).reshape(-1))
           for x in ora.run_game(6, 3, row, col, wt, att, ora.standard_reach(row, att)).lists()]
    g = geq.GameGraph.from_csr(row, col, wt, att, geq.EnergyConf.STANDARD)
    empty = geq.GameGraph.empty(geq.EnergyConf.STANDARD)
    got = [geq.run_batch_raw([g], ctx)[:2], geq.run_batch_raw([g, empty], ctx)[:2]]
    got = [(o[0], d[0]) for o, d in got] + [geq.run_static(g, ctx)[:2]]
    with Server(ctx) as srv:
        for t in [srv.submit(g) for _ in range(3)]:
            got.append(srv.poll(t)[:2])
    for o, d in got:
        o = np.asarray(o).astype(np.int64)
        for v, x in enumerate(exp):
            assert np.array_equal(np.sort(d[o[v]:o[v + 1]]), x), f"position {v}"
