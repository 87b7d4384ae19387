"""The two forms of a worklist round -- positions spread over all warps (small
frontiers) and 32 positions per warp (large ones) -- give the same lists: a
game solved alone against many disjoint copies of it solved as one game, whose
frontiers are large.  Sizes sit at the limits of the lane
path: up to 18 successors (16 stay in it), initial lists of up to 20 energies
(16 stay in it), updates with several merges, single-successor defenders."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from helpers import canon
from oracle import ora

pytestmark = pytest.mark.gpu

N_EL = 6


@pytest.fixture(scope="module")
def geq():
    import gpuequiv_b200 as geq
    return geq


@pytest.fixture(scope="module")
def ctx(geq):
    c = geq.Context(0)
    yield c
    c.close()


def make_game(seed, n, mean_deg, merges):
    """A bipartite game (positions of one kind point at the other) with
    initial lists at a tenth of the attackers."""
    rng = np.random.default_rng(seed)
    att = (rng.random(n) < 0.55).astype(np.uint8)
    att[:2] = (1, 0)
    deg = np.minimum(rng.geometric(1.0 / mean_deg, n), 18).astype(np.int64) - (rng.random(n) < 0.15)
    row = np.zeros(n + 1, np.uint32)
    np.cumsum(deg, out=row[1:])
    m = int(row[-1])
    A, D = np.nonzero(att)[0].astype(np.uint32), np.nonzero(att == 0)[0].astype(np.uint32)
    src_att = np.repeat(att, deg).astype(bool)
    col = np.where(src_att, D[rng.integers(0, len(D), m)], A[rng.integers(0, len(A), m)]).astype(np.uint32)
    wt = np.zeros(m, np.uint32)
    for k in range(merges):  # a component in some of the elements
        pos = rng.integers(0, N_EL, m)
        code = np.where(rng.random(m) < 0.5, 1, rng.integers(2, N_EL + 2, m))
        code = np.where(code == pos + 2, 1, code).astype(np.uint32)
        use = rng.random(m) < 0.6 / (k + 1)
        wt = np.where(use, (wt & ~(np.uint32(15) << (4 * pos).astype(np.uint32)))
                      | (code << (4 * pos).astype(np.uint32)), wt).astype(np.uint32)
    counts = np.zeros(n, np.int64)
    pick = A[rng.random(len(A)) < 0.1]
    counts[pick] = rng.integers(1, 21, len(pick))
    sinks = np.nonzero((att == 0) & (deg == 0))[0]
    counts[sinks] = 1
    offs = np.zeros(n + 1, np.uint64)
    offs[1:] = np.cumsum(counts)
    data = rng.integers(0, 1 << 12, int(offs[-1])).astype(np.uint32)
    data[offs[sinks].astype(np.int64)] = 0
    return row, col, wt, att, offs, data, np.concatenate([sinks, pick]).astype(np.uint32)


def copies(game, k):
    row, col, wt, att, offs, data, reach = game
    n, m, t = len(att), len(col), len(data)
    base = np.arange(k, dtype=np.uint64)
    rows = (row[:-1][None, :] + (base * m).astype(np.uint32)[:, None]).reshape(-1)
    off = (offs[:-1][None, :] + (base * t)[:, None]).reshape(-1)
    shift = (base * n).astype(np.uint32)[:, None]
    return (np.append(rows, np.uint32(k * m)), (col[None, :] + shift).reshape(-1), np.tile(wt, k), np.tile(att, k),
            np.append(off, np.uint64(k * t)), np.tile(data, k), (reach[None, :] + shift).reshape(-1))


def solve(geq, ctx, game):
    from gpuequiv_b200._lib import check, geq_energy_lists, lib
    row, col, wt, att, offs, data, reach = game
    g = geq.GameGraph.from_csr(row, col, wt, att, geq.EnergyConf.STANDARD)
    view = g.c_view()
    init = geq_energy_lists(len(att), 1, offs.ctypes.data_as(C.POINTER(C.c_uint64)),
                            data.ctypes.data_as(C.POINTER(C.c_uint32)))
    reach = np.ascontiguousarray(reach)
    sol, out = C.c_void_p(), geq_energy_lists()
    check(lib.geq_energy_game_run(ctx.h, C.byref(view), C.byref(init), reach.ctypes.data_as(C.POINTER(C.c_uint32)),
                                  len(reach), C.byref(sol)))
    check(lib.geq_solution_lists(sol, 0, C.byref(out)))
    o = np.ctypeslib.as_array(out.offsets, shape=(len(att) + 1,)).copy()
    d = np.ctypeslib.as_array(out.data, shape=(int(o[-1]),)).copy()
    lib.geq_solution_free(sol)
    return o, d


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 255, 256, 257, 400, 401, 4096, 4097, 32768, 32769])
@pytest.mark.parametrize("form", ["run", "batch", "static"])
def test_launch_forms(geq, ctx, n, form):
    """Sizes at the lines between one block, a cluster and graphs of rounds,
    through the calls that take them: one game (a launch of its own up to
    32,768 positions), the same game beside an empty one (an upload and rounds),
    and the allocation-free call."""
    row, col, wt, att, _, _, _ = make_game(100 + n, max(n, 2), 2.5, 1)
    if n == 1:
        row, col, wt, att = row[:2] * 0, col[:0], wt[:0], att[1:]
    g = geq.GameGraph.from_csr(row, col, wt, att, geq.EnergyConf.STANDARD)
    if form == "static":
        o, d, _ = geq.run_static(g, ctx)
    elif form == "run":
        offs, data, _ = geq.run_batch_raw([g], ctx)
        o, d = offs[0], data[0]
    else:
        offs, data, _ = geq.run_batch_raw([g, geq.GameGraph.empty(geq.EnergyConf.STANDARD)], ctx)
        o, d = offs[0], data[0]
    exp = ora.run_game(6, 3, row, col, wt, att, ora.standard_reach(row, att)).lists()
    for v in range(len(att)):
        assert canon(d[int(o[v]):int(o[v + 1])]) == canon(exp[v]), f"position {v}"


@pytest.mark.parametrize("n", [30_000, 60_000])
@pytest.mark.parametrize("indeg", [63, 64, 511, 512, 513, 20_000])
def test_long_predecessor_lists(geq, ctx, n, indeg):
    """Positions with as many predecessors as the lines between the ways to
    push them, many of them side by side, inside one launch (30,000 positions)
    and as rounds of kernels (60,000)."""
    rng = np.random.default_rng(indeg)
    hubs = 12  # defenders without successors, each reached by `indeg` attackers
    srcs = np.concatenate([np.sort(rng.choice(np.arange(hubs, n), indeg, replace=False)) for _ in range(hubs)])
    dst = np.repeat(np.arange(hubs), indeg)
    extra_s = np.arange(hubs, n)  # and a chain, so that the pushes go on
    src = np.concatenate([srcs, extra_s]).astype(np.int64)
    dst = np.concatenate([dst, np.concatenate([extra_s[1:], [hubs]])])
    order = np.argsort(src, kind="stable")
    src, dst = src[order], dst[order].astype(np.uint32)
    row = np.zeros(n + 1, np.uint32)
    row[1:] = np.cumsum(np.bincount(src, minlength=n))
    wt = (np.uint32(1) << (4 * rng.integers(0, N_EL, len(src))).astype(np.uint32)).astype(np.uint32)
    att = np.ones(n, np.uint8)
    att[:hubs] = 0
    g = geq.GameGraph.from_csr(row, dst, wt, att, geq.EnergyConf.STANDARD)
    offs, data, _ = geq.run_batch_raw([g], ctx)
    o, d = offs[0].astype(np.int64), data[0]
    exp = ora.run_game(6, 3, row, dst, wt, att, ora.standard_reach(row, att))
    lists = exp.lists()
    assert np.array_equal(np.diff(o), [len(x) for x in lists])
    for v in range(n):
        assert canon(d[o[v]:o[v + 1]]) == canon(lists[v]), f"position {v}"


@pytest.mark.parametrize("seed,n,mean_deg,merges", [(1, 6000, 3.0, 1), (2, 9000, 1.6, 2), (3, 5000, 7.0, 3),
                                                    (4, 7000, 2.5, 0)])
def test_small_and_large_rounds_agree(geq, ctx, seed, n, mean_deg, merges):
    game = make_game(seed, n, mean_deg, merges)
    o, d = solve(geq, ctx, game)
    row, col, wt, att, offs, data, reach = game
    exp = ora.run_game(6, 3, row, col, wt, att, reach, init=(offs, data)).lists()
    for v in range(n):
        assert canon(d[int(o[v]):int(o[v + 1])]) == canon(exp[v]), f"position {v}"
    k = 320_000 // n
    ob, db = solve(geq, ctx, copies(game, k))
    cnt = np.diff(o.astype(np.int64))
    assert np.array_equal(np.diff(ob.astype(np.int64)), np.tile(cnt, k))
    # lists are sets: compared sorted, position by position
    exp_d = d[np.lexsort((d, np.repeat(np.arange(n), cnt)))]
    got_d = db[np.lexsort((db, np.repeat(np.arange(k * n), np.tile(cnt, k))))]
    assert np.array_equal(got_d, np.tile(exp_d, k))
