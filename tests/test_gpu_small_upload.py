"""Uploads at the line (8,192 positions) between one launch for checks, reverse
edges and restart, and launches of their own: standard starts, given lists and
positions to reach, several games to an upload, solved again and again; what is
refused on one side is refused on the other.  Selections at the line (4,096
positions) between one launch and a scan."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from helpers import canon
from oracle import ora
from test_gpu_rounds import make_game

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 33, 512, 4095, 8191, 8192, 8193]


@pytest.fixture(scope="module")
def geq():
    import gpuequiv_b200 as geq
    return geq


@pytest.fixture(scope="module")
def ctx(geq):
    c = geq.Context(0)
    yield c
    c.close()


def same(o, d, exp):
    for v in range(len(exp)):
        assert canon(d[int(o[v]):int(o[v + 1])]) == canon(exp[v]), f"position {v}"


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("parts", [1, 3])
def test_resident(geq, ctx, n, parts):
    """`n` positions in all, in `parts` games, solved three times."""
    cuts = [n * k // parts for k in range(parts + 1)]
    games = []
    for k in range(parts):
        m = cuts[k + 1] - cuts[k]
        row, col, wt, att = make_game(7 * n + k, max(m, 2), 2.5, 2)[:4]
        if m < 2:
            row, col, wt, att = np.zeros(m + 1, np.uint32), col[:0], wt[:0], np.zeros(m, np.uint8)
        games.append((row, col, wt, att))
    dg = geq.DeviceGames([geq.GameGraph.from_csr(*g, geq.EnergyConf.STANDARD) for g in games], ctx)
    exp = [ora.run_game(6, 3, *g, ora.standard_reach(g[0], g[3])).lists() if len(g[3]) else [] for g in games]
    for _ in range(3):
        dg.solve()
        offs, data = dg.download_raw()[:2]
        for k in range(parts):
            same(offs[k], data[k], exp[k])
    dg.close()


@pytest.mark.parametrize("n", [s for s in SIZES if s > 30])
def test_initial_lists(geq, ctx, n):
    from gpuequiv_b200._lib import check, geq_energy_lists, geq_game_graph, lib
    row, col, wt, att, offs, data, reach = make_game(11 * n, n, 2.2, 2)
    view = (geq_game_graph * 1)(geq.GameGraph.from_csr(row, col, wt, att, geq.EnergyConf.STANDARD).c_view())
    init = geq_energy_lists(n, 1, offs.ctypes.data_as(C.POINTER(C.c_uint64)),
                            data.ctypes.data_as(C.POINTER(C.c_uint32)))
    ip = (C.POINTER(geq_energy_lists) * 1)(C.pointer(init))
    rp = (C.POINTER(C.c_uint32) * 1)(reach.ctypes.data_as(C.POINTER(C.c_uint32)))
    nr = (C.c_uint32 * 1)(len(reach))
    h = C.c_void_p()
    check(lib.geq_device_games_create(ctx.h, 1, view, ip, rp, nr, C.byref(h)))
    exp = ora.run_game(6, 3, row, col, wt, att, reach, init=(offs, data)).lists()
    for _ in range(2):
        check(lib.geq_device_games_solve(ctx.h, h, None))
        sol, out = C.c_void_p(), geq_energy_lists()
        check(lib.geq_device_games_download(ctx.h, h, C.byref(sol)))
        check(lib.geq_solution_lists(sol, 0, C.byref(out)))
        o = np.ctypeslib.as_array(out.offsets, shape=(n + 1,)).copy()
        d = np.ctypeslib.as_array(out.data, shape=(max(int(o[-1]), 1),)).copy()
        lib.geq_solution_free(sol)
        same(o, d, exp)
    lib.geq_device_games_free(h)


@pytest.mark.parametrize("n", [100, 8192, 8193])
@pytest.mark.parametrize("bad", ["column", "update"])
def test_refused(geq, ctx, n, bad):
    """An invalid upload is an error on both sides of the line, and the next
    valid one is solved."""
    row, col, wt, att = make_game(n, n, 2.5, 1)[:4]
    good = geq.GameGraph.from_csr(row, col, wt, att, geq.EnergyConf.STANDARD)
    c2, w2 = col.copy(), wt.copy()
    if bad == "column":
        c2[-1] = n
    else:
        w2[-1] = 8
    with pytest.raises(geq.GeqError) as e:
        geq.DeviceGames([geq.GameGraph.from_csr(row, c2, w2, att, geq.EnergyConf.STANDARD)], ctx)
    assert e.value.name == "INVALID_INPUT"
    dg = geq.DeviceGames([good], ctx)
    dg.solve()
    offs, data = dg.download_raw()[:2]
    same(offs[0], data[0], ora.run_game(6, 3, row, col, wt, att, ora.standard_reach(row, att)).lists())
    dg.close()


@pytest.mark.parametrize("n_jobs", [4095, 4096, 4097])
def test_selection(geq, ctx, n_jobs):
    rng = np.random.default_rng(n_jobs)
    edges = zip(rng.integers(0, 9, 16).tolist(), rng.integers(0, 9, 16).tolist(), rng.integers(0, 2, 16).tolist())
    lts = geq.TransitionSystem(list(edges) + [(0, 8, 0)])
    pairs = [(p, q) for p in range(9) for q in range(9)]
    few = geq.compare_batch([(lts, p, q) for p, q in pairs], ctx, minimize=False)
    many = geq.compare_batch([(lts, *pairs[i % len(pairs)]) for i in range(n_jobs)], ctx, minimize=False)
    for i, got in enumerate(many):
        assert canon(got.array) == canon(few[i % len(pairs)].array), i
