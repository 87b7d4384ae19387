"""The forms of the multi-word solver's rounds against the oracle: antichains
in shared memory (energies of one, two and four words) up to, at and beyond
their 256 members, other energy sizes in the warps' scratch, games whose rounds
run inside launches of a cluster (up to 8,192 positions) or of the whole device
(up to 262,144) and larger ones."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from helpers import canon
from oracle import ora

pytestmark = pytest.mark.gpu

CONFS = [(2, 65535), (3, 1000), (30, 3), (50, 3), (1, 0xFFFFFFFF), (5, 0xFFFFFFFF)]


@pytest.fixture(scope="module")
def geq():
    import gpuequiv_b200 as geq
    return geq


@pytest.fixture(scope="module")
def ctx(geq):
    c = geq.Context(0)
    yield c
    c.close()


def pack(geq, conf, values):
    c = geq.EnergyConf(*conf)
    out = np.zeros((len(values), c.energy_size()), np.uint32)
    per = 32 // c.energy_bits()
    for i in range(conf[0]):
        shift = np.uint32(c.energy_bits() * (i % per))
        out[:, i // per] |= values[:, i].astype(np.uint32) << shift
    return out


def update_words(geq, conf, codes):
    c = geq.EnergyConf(*conf)
    out = np.zeros((len(codes), c.update_size()), np.uint32)
    per = 32 // c.update_bits()
    for i in range(conf[0]):
        out[:, i // per] |= codes[:, i].astype(np.uint32) << np.uint32(c.update_bits() * (i % per))
    return out


def run_both(geq, ctx, conf, row, col, wt, att, reach, offs, data):
    from gpuequiv_b200._lib import check, geq_energy_lists, lib
    cf = geq.EnergyConf(*conf)
    es = cf.energy_size()
    g = geq.GameGraph.from_csr(row, col, wt, att, cf)
    view = g.c_view()
    flat = np.ascontiguousarray(data.reshape(-1)) if data.size else np.zeros(1, np.uint32)
    init = geq_energy_lists(len(att), es, offs.ctypes.data_as(C.POINTER(C.c_uint64)),
                            flat.ctypes.data_as(C.POINTER(C.c_uint32)))
    sol, out = C.c_void_p(), geq_energy_lists()
    check(lib.geq_energy_game_run(ctx.h, C.byref(view), C.byref(init), reach.ctypes.data_as(C.POINTER(C.c_uint32)),
                                  len(reach), C.byref(sol)))
    check(lib.geq_solution_lists(sol, 0, C.byref(out)))
    o = np.ctypeslib.as_array(out.offsets, shape=(len(att) + 1,)).astype(np.int64)
    d = (np.ctypeslib.as_array(out.data, shape=(int(o[-1]) * es,)).copy() if o[-1] else
         np.zeros(0, np.uint32)).reshape(-1, es)
    lib.geq_solution_free(sol)
    exp = ora.run_game(conf[0], conf[1], row, col, np.asarray(wt).reshape(-1), att, reach, init=(offs, flat)).lists()
    assert np.array_equal(np.diff(o), [len(x) for x in exp])
    for v in range(len(att)):
        assert canon(d[o[v]:o[v + 1]]) == canon(exp[v]), f"position {v}"


@pytest.mark.parametrize("conf", CONFS)
@pytest.mark.parametrize("members", [1, 31, 32, 33, 255, 256, 257, 300])
def test_antichain_sizes(geq, ctx, conf, members):
    """0 (attacker) -> 1 (defender) -> 2 and 3 (attackers with given lists of
    `members` energies); 4 (defender, one successor) -> 2; 0 -> 4."""
    rng = np.random.default_rng(members)
    el, mx = conf
    lists = []
    for _ in range(2):
        v = rng.integers(0, min(mx, 3) + 1, (members, el)).astype(np.uint64)
        if el > 1 and mx >= 300:  # an antichain: one element up, another down
            v[:, 0] = np.arange(members)
            v[:, 1] = members - np.arange(members)
        lists.append(pack(geq, conf, v))
    if members >= 255:  # keep the product of the two lists small
        lists[1] = lists[1][:2]
    row = np.array([0, 2, 4, 4, 4, 5], np.uint32)
    col = np.array([1, 4, 2, 3, 2], np.uint32)
    codes = np.zeros((5, el), np.uint32)
    codes[0, 0] = 1
    codes[2, el - 1] = 1
    if el > 2:
        codes[3, 1] = 2 + 2
        codes[4, 2] = 1
    offs = np.array([0, 0, 0, len(lists[0]), len(lists[0]) + len(lists[1]), len(lists[0]) + len(lists[1])], np.uint64)
    run_both(geq, ctx, conf, row, col, update_words(geq, conf, codes), np.array([1, 0, 1, 1, 0], np.uint8),
             np.array([2, 3], np.uint32), offs, np.concatenate(lists))


@pytest.mark.parametrize("conf", [(30, 3), (1, 0xFFFFFFFF)])
@pytest.mark.parametrize("n", [1, 33, 8192, 8193, 65536, 65537, 262144, 262145])
def test_game_sizes(geq, ctx, conf, n):
    rng = np.random.default_rng(n)
    att = (rng.random(n) < 0.6).astype(np.uint8)
    deg = rng.integers(0, 3, n)
    row = np.zeros(n + 1, np.uint32)
    row[1:] = np.cumsum(deg)
    m = int(row[-1])
    col = rng.integers(0, n, m).astype(np.uint32)
    codes = np.zeros((m, conf[0]), np.uint32)
    codes[np.arange(m), rng.integers(0, conf[0], m)] = rng.random(m) < 0.2
    reach = np.nonzero((att == 0) & (deg == 0))[0].astype(np.uint32)
    offs = np.zeros(n + 1, np.uint64)
    offs[1:] = np.cumsum((att == 0) & (deg == 0))
    es = geq.EnergyConf(*conf).energy_size()
    run_both(geq, ctx, conf, row, col, update_words(geq, conf, codes), att, reach, offs,
             np.zeros((int(offs[-1]), es), np.uint32))


@pytest.mark.parametrize("conf", [(2, 65535), (30, 3), (50, 3), (1, 0xFFFFFFFF)])
@pytest.mark.parametrize("na,nb", [(1, 1), (1, 40), (40, 1), (5, 7), (31, 33), (33, 32), (2, 128)])
def test_suprema_left_out(geq, ctx, conf, na, nb):
    """A defender over lists that share members, hold energies above and below
    the other's, and none comparable: products of which most, some or no
    suprema are left out before they are inserted."""
    rng = np.random.default_rng(1000 * na + nb)
    el, mx = conf
    top = min(mx, 3)
    for kind in ("shared", "above", "apart"):
        a = rng.integers(0, top + 1, (na, el)).astype(np.uint64)
        b = rng.integers(0, top + 1, (nb, el)).astype(np.uint64)
        k = min(na, nb)
        if kind == "shared":
            b[:k:2] = a[:k:2]
        elif kind == "above":  # every second energy above or below one of the other list
            b[:k:4] = np.minimum(a[:k:4] + rng.integers(0, 2, a[:k:4].shape).astype(np.uint64), top)
            a[2:k:4] = np.minimum(b[2:k:4] + rng.integers(0, 2, b[2:k:4].shape).astype(np.uint64), top)
        lists = [pack(geq, conf, a), pack(geq, conf, b)]
        row = np.array([0, 1, 3, 3, 3], np.uint32)
        col = np.array([1, 2, 3], np.uint32)
        offs = np.array([0, 0, 0, na, na + nb], np.uint64)
        run_both(geq, ctx, conf, row, col, update_words(geq, conf, np.zeros((3, el), np.uint32)),
                 np.array([1, 0, 1, 1], np.uint8), np.array([2, 3], np.uint32), offs, np.concatenate(lists))
