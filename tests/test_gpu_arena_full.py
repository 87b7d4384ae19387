"""Rounds inside one launch whose results outgrow the energy arena: the launch is
left, the host compacts and the rounds go on -- in cluster launches of small
uploads, in those of larger uploads with small frontiers, from a lone game's
launch to the general path, and in the multi-word solver's cluster and
cooperative launches."""
from __future__ import annotations

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


def layers(geq, conf, width, depth, tail):
    """Attackers of layer k reach layer k-1 by a decrement of each of the `el`
    elements (so all of a layer have the same list), then `tail` layers of
    defenders and attackers with one successor each that hold copies."""
    c, el = geq.EnergyConf(*conf), conf[0]
    n0, n = width * (depth + 1), width * (depth + 1 + tail)
    att = np.ones(n, np.uint8)
    att[:width] = 0
    for t in range(0, tail, 2):
        att[n0 + t * width:n0 + (t + 1) * width] = 0
    deg = np.concatenate([np.zeros(width), np.full(n0 - width, el), np.ones(n - n0)]).astype(np.int64)
    row = np.zeros(n + 1, np.uint32)
    np.cumsum(deg, out=row[1:])
    rng = np.random.default_rng(width)
    col = np.concatenate([np.repeat(np.arange(depth) * width, width * el) + rng.integers(0, width, width * depth * el),
                          np.arange(n0, n) - width]).astype(np.uint32)
    wt = np.zeros((len(col), c.update_size()), np.uint32)
    k, i, per = np.arange(width * depth * el), np.tile(np.arange(el), width * depth), 32 // c.update_bits()
    wt[k, i // per] = np.uint32(1) << (c.update_bits() * (i % per)).astype(np.uint32)
    return row, col, wt, att


def check(geq, conf, width, depth, tail, graphs, ctx, compactions):
    offs, data, stats = geq.run_batch_raw(graphs, ctx)
    assert stats["arena_compactions"] >= compactions
    o = offs[0].astype(np.int64)
    es = geq.EnergyConf(*conf).energy_size()
    d = data[0].reshape(-1, es)
    row, col, wt, att = layers(geq, conf, 1, depth, tail)
    exp = ora.run_game(conf[0], conf[1], row, col, wt.reshape(-1), att, np.array([0], np.uint32)).lists()
    order = lambda x: x[np.lexsort(x.T)]
    for k in range(depth + 1 + tail):
        want = order(np.asarray(exp[k], np.uint32).reshape(-1, es))
        lens = np.diff(o)[k * width:(k + 1) * width]
        assert (lens == len(want)).all(), f"layer {k}"
        for v in range(k * width, (k + 1) * width):
            assert np.array_equal(order(d[o[v]:o[v + 1]]), want), f"position {v}"


@pytest.mark.parametrize("tail,form", [(8, "run"), (8, "batch"), (20, "run"), (20, "batch")])
def test_one_word(geq, ctx, tail, form):
    """22,100 positions (all rounds in cluster launches) and 42,500 (those of at
    most 2,048 positions): 1,700 lists of 330 energies a round, an arena of 4
    million words."""
    conf = (8, 4)
    g = geq.GameGraph.from_csr(*layers(geq, conf, 1700, 4, tail), geq.EnergyConf(*conf))
    graphs = [g] + [geq.GameGraph.empty(geq.EnergyConf(*conf))] * (form == "batch")
    check(geq, conf, 1700, 4, tail, graphs, ctx, 1)


@pytest.mark.parametrize("width", [200, 600])
def test_two_words(geq, ctx, width):
    """3,400 positions (a cluster) and 10,200 (every SM), lists of up to 165
    energies, an arena of 16 energies per position and edge."""
    conf = (4, 1000)
    g = geq.GameGraph.from_csr(*layers(geq, conf, width, 8, 8), geq.EnergyConf(*conf))
    check(geq, conf, width, 8, 8, [g], ctx, 1)
