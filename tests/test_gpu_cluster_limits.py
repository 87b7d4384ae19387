"""Where rounds leave the launches of one cluster (16 of the SMs) for kernels
over the whole device: games with many edges, and rounds with more than 1,792
positions that take a warp each."""
from __future__ import annotations

import time

import numpy as np
import pytest

from helpers import canon
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


def dense_game(n, m, seed=1):
    """Exactly m edges: a tenth of the defenders have no successors, the others
    one to three; the attackers have the rest."""
    rng = np.random.default_rng(seed)
    att = (np.arange(n) % 5 < 3).astype(np.uint8)
    A, D = np.nonzero(att)[0], np.nonzero(att == 0)[0]
    few = np.repeat(D[len(D) // 10:], rng.integers(1, 4, len(D) - len(D) // 10))
    src = np.sort(np.concatenate([few, A[rng.integers(0, len(A), m - len(few))]]))
    row = np.zeros(n + 1, np.uint32)
    np.cumsum(np.bincount(src, minlength=n), out=row[1:])
    col = np.where(att[src] == 1, D[rng.integers(0, len(D), m)], A[rng.integers(0, len(A), m)]).astype(np.uint32)
    wt = np.where(rng.random(m) < 0.3, np.uint32(1) << (4 * rng.integers(0, 6, m)).astype(np.uint32), 0)
    return row, col, wt.astype(np.uint32), att


def layers(width, depth):
    """Attackers of layer k reach layer k-1 by a decrement of each element, so
    all of a layer have the same list: 1, 6, 21, 56, 96, ... energies."""
    n = width * (depth + 1)
    att = np.ones(n, np.uint8)
    att[:width] = 0
    deg = np.full(n, 6)
    deg[:width] = 0
    row = np.zeros(n + 1, np.uint32)
    np.cumsum(deg, out=row[1:])
    rng = np.random.default_rng(5)
    col = np.repeat(np.arange(depth) * width, width * 6) + rng.integers(0, width, width * depth * 6)
    wt = np.tile(np.uint32(1) << (4 * np.arange(6)).astype(np.uint32), width * depth)
    return row, col.astype(np.uint32), wt.astype(np.uint32), att


def seconds(call):
    t0 = time.perf_counter()
    call()
    return time.perf_counter() - t0


def solve(geq, ctx, g, form):
    graphs = [geq.GameGraph.from_csr(*g, geq.EnergyConf.STANDARD)]
    if form == "batch":
        graphs.append(geq.GameGraph.empty(geq.EnergyConf.STANDARD))
    offs, data, stats = geq.run_batch_raw(graphs, ctx)
    return offs[0].astype(np.int64), data[0], stats


@pytest.mark.parametrize("form", ["run", "batch"])
@pytest.mark.parametrize("n,m", [(2500, 196608), (2500, 196609), (9000, 196608), (9000, 196609), (700, 300000)])
def test_edges(geq, ctx, n, m, form):
    g = dense_game(n, m)
    o, d, stats = solve(geq, ctx, g, form)
    if m > 196608:  # every round by the four kernels
        assert stats["kernel_launches"] >= 4 * stats["rounds"]
    exp = ora.run_game(6, 3, *g, ora.standard_reach(g[0], g[3])).lists()
    for v in range(n):
        assert canon(d[o[v]:o[v + 1]]) == canon(exp[v]), f"position {v}"


@pytest.mark.parametrize("form", ["run", "batch"])
@pytest.mark.parametrize("width", [1792, 1793, 3000])
def test_large_positions(geq, ctx, width, form):
    """Layers of `width` positions whose lists leave the lane path from the
    second layer on."""
    depth = 6
    g = layers(width, depth)
    o, d, stats = solve(geq, ctx, g, form)
    if width > 1792:
        assert stats["kernel_launches"] >= 4 * (depth - 3)
    g1 = layers(1, depth)
    exp = ora.run_game(6, 3, *g1, ora.standard_reach(g1[0], g1[3])).lists()
    for k in range(depth + 1):
        want = np.sort(np.asarray(exp[k]).reshape(-1)).astype(np.uint32)
        lens = np.diff(o)[k * width:(k + 1) * width]
        assert (lens == len(want)).all(), f"layer {k}"
        got = np.sort(d[o[k * width]:o[(k + 1) * width]].reshape(width, len(want)), axis=1)
        assert (got == want).all(), f"layer {k}"


@pytest.mark.parametrize("m", [4096, 4097, 65536, 160000])
def test_few_positions_many_edges(geq, ctx, m):
    """400 positions in one block up to 4,096 edges, in a cluster above; alone
    a game is not slower than beside an empty one (an upload and its rounds)."""
    g = dense_game(400, m, seed=3)
    o, d, _ = solve(geq, ctx, g, "run")
    exp = ora.run_game(6, 3, *g, ora.standard_reach(g[0], g[3])).lists()
    for v in range(400):
        assert canon(d[o[v]:o[v + 1]]) == canon(exp[v]), f"position {v}"
    if m > 65536:  # whole calls: a game alone is uploaded inside its launch
        alone = min(seconds(lambda: solve(geq, ctx, g, "run")) for _ in range(5))
        beside = min(seconds(lambda: solve(geq, ctx, g, "batch")) for _ in range(5))
        assert alone < 1.5 * beside, (alone, beside)


@pytest.mark.parametrize("n,width", [(3000, 1), (3000, 16), (3000, 17), (20000, 1), (20000, 16)])
def test_rounds_of_few_positions(geq, ctx, n, width):
    """Chains side by side, joined at their ends: rounds of `width` positions,
    which block 0 runs alone up to 16, between wider ones."""
    k = n // width
    at = np.arange(k * width).reshape(width, k)  # chain j: at[j, 0] (a sink) <- at[j, 1] <- ...
    att = np.tile((np.arange(k) % 3 != 0).astype(np.uint8), width)
    src = [at[:, 1:].reshape(-1)]
    dst = [at[:, :-1].reshape(-1)]
    # a fan of 40 attackers over the chains' ends and of 40 more over those
    fan = k * width + np.arange(80)
    src += [np.repeat(fan[:40], width), np.repeat(fan[40:], 2)]
    dst += [np.tile(at[:, -1], 40), fan[:40][(np.arange(80) * 7) % 40]]
    att = np.append(att, np.ones(80, np.uint8))
    src, dst = np.concatenate(src), np.concatenate(dst)
    order = np.argsort(src, kind="stable")
    src, dst = src[order], dst[order].astype(np.uint32)
    row = np.zeros(len(att) + 1, np.uint32)
    np.cumsum(np.bincount(src, minlength=len(att)), out=row[1:])
    rng = np.random.default_rng(n + width)
    wt = np.where(rng.random(len(src)) < 0.01, np.uint32(1) << (4 * rng.integers(0, 6, len(src))).astype(np.uint32), 0)
    g = (row, dst, wt.astype(np.uint32), att)
    exp = ora.run_game(6, 3, *g, ora.standard_reach(row, att)).lists()
    for form in ("run", "batch"):
        o, d, stats = solve(geq, ctx, g, form)
        assert stats["rounds"] >= k
        for v in range(len(att)):
            assert canon(d[o[v]:o[v + 1]]) == canon(exp[v]), f"position {v}"


def test_chain_time(geq, ctx):
    """A chain alone (a cluster) against the call that is always one block."""
    n = 4000
    row = np.minimum(np.arange(n + 1), n - 1).astype(np.uint32)
    att = np.tile(np.array([1, 0], np.uint8), n // 2)
    g = geq.GameGraph.from_csr(row, np.arange(1, n, dtype=np.uint32), np.zeros(n - 1, np.uint32), att,
                               geq.EnergyConf.STANDARD)
    alone = min(seconds(lambda: geq.run_batch_raw([g], ctx)) for _ in range(5))
    block = min(seconds(lambda: geq.run_static(g, ctx)) for _ in range(5))
    assert alone < 1.25 * block, (alone, block)


def test_two_large_positions_a_round(geq, ctx):
    """Two positions a round take as long as one: each has a warp."""
    conf = geq.EnergyConf(8, 4)

    def call(width):
        depth = 5
        row = np.concatenate([np.zeros(width), np.arange(width * depth + 1) * 8]).astype(np.uint32)
        col = np.repeat(np.arange(depth * width), 8).astype(np.uint32)
        wt = np.tile(np.uint32(1) << (4 * np.arange(8)).astype(np.uint32), width * depth).astype(np.uint32)
        att = (np.arange(width * (depth + 1)) >= width).astype(np.uint8)
        g = geq.GameGraph.from_csr(row, col, wt, att, conf)
        empty = geq.GameGraph.empty(conf)
        return [min(seconds(lambda: geq.run_batch_raw(gs, ctx)) for _ in range(4)) for gs in ([g], [g, empty])]

    for one, two in zip(call(1), call(2)):
        assert two < 1.4 * one, (one, two)
