"""The work that the solver's speed is measured on.

Every case goes through the public entry points with the inputs a host
program has in hand: game graphs or transition systems in host memory, a
context, and where a program would keep one, games resident on the device or a
running server.  All inputs are synthetic and come from the generators of
``gpuequiv_b200.synth``; the jobs of the batched configuration are its recorded
seeds (``data/batched_seeds.json``), whose games have between 6 and 200,000
positions.  The seed renumbers states, labels and positions of the recorded jobs
and generated games, so that every seed gives other inputs of one size.
"""
from __future__ import annotations

import ctypes as C
import functools
import math
from concurrent.futures import ThreadPoolExecutor

import numpy as np

import gpuequiv_b200 as geq
from gpuequiv_b200 import synth
from gpuequiv_b200._lib import check, lib
from gpuequiv_b200.serving import Server

_ROWS = sorted((int(r[1]), int(r[0]), int(r[2])) for r in synth.batched_manifest()["jobs"])
_POS = np.array([r[0] for r in _ROWS], dtype=np.int64)
_EDGES = np.array([r[2] for r in _ROWS], dtype=np.int64)

# relations asked of a whole system
_RELATIONS = ("enabledness", "traces", "failures", "simulation", "bisimulation")
# energies of a compare query's table (the longest list of the batched configuration has fewer)
_WIDTH = 256


def listed():
    return [
        # one call of EnergyGame::run on a game as small as most of the batched configuration's
        {"name": "game_tiny", "kind": "game", "positions": 80},
        # the same on a game of a few thousand positions (a query on a 100-state system)
        {"name": "game_small", "kind": "game", "positions": 2500},
        # one larger game per call: more positions than one block takes
        {"name": "game_medium", "kind": "game", "positions": 42000},
        # the batched configuration from host buffers: uneven games, lists back on the host
        {"name": "batch_host", "kind": "batch", "games": 512, "max_positions": 200000, "resident": False},
        # games kept on the device and solved again, as an autotuner or a what-if loop does
        {"name": "batch_resident", "kind": "batch", "games": 1400, "max_positions": 200000, "resident": True},
        # the energy-game-only stress configuration, at its full size
        {"name": "stress_full", "kind": "stress", "positions": 2000000, "edges": 10000000},
        # an energy of two words, solved by the multi-word path
        {"name": "wide_two_words", "kind": "wide", "elements": 30, "max": 3, "positions": 12000},
        # equivalence queries as they come, one call each
        {"name": "compare_each", "kind": "compare", "jobs": 12, "max_positions": 20000, "together": False},
        # many equivalence queries at once: minimisation, game construction and solving of all
        {"name": "compare_batch", "kind": "compare", "jobs": 512, "max_positions": 200000, "together": True},
        # all pairs of a small system (the small configuration)
        {"name": "equivalences_small", "kind": "equivalences", "states": 40, "transitions": 120, "family": "small"},
        # all pairs of a larger system (the generator of the large configuration)
        {"name": "equivalences_large", "kind": "equivalences", "states": 3000, "transitions": 12000,
         "family": "large"},
        # a burst of requests to the serving loop, answered in order
        {"name": "serve_burst", "kind": "serve", "games": 256, "max_positions": 30000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["game", "game", "batch", "stress", "wide", "compare", "compare", "equivalences", "serve"])
    if kind == "game":
        return {"kind": "game", "positions": _log(rng, 40, 150000)}
    if kind == "batch":
        return {"kind": "batch", "games": _log(rng, 3, 600), "max_positions": _log(rng, 2000, 200000),
                "resident": rng.random() < 0.5}
    if kind == "stress":
        n = _log(rng, 3000, 1500000)
        return {"kind": "stress", "positions": n, "edges": int(n * rng.uniform(2.5, 5.0))}
    if kind == "wide":
        el, mx = rng.choice([(30, 3), (16, 7), (3, 1000), (1, 0xFFFFFFFF)])
        return {"kind": "wide", "elements": el, "max": mx, "positions": _log(rng, 300, 20000)}
    if kind == "compare":
        together = rng.random() < 0.5
        return {"kind": "compare", "jobs": _log(rng, 16, 480) if together else rng.randint(12, 24),
                "max_positions": _log(rng, 3000, 200000 if together else 60000), "together": together}
    if kind == "equivalences":
        if rng.random() < 0.5:
            n = rng.randint(16, 44)
            return {"kind": "equivalences", "states": n, "transitions": int(n * rng.uniform(2.0, 3.0)),
                    "family": "small"}
        n = _log(rng, 300, 3000)
        return {"kind": "equivalences", "states": n, "transitions": 4 * n, "family": "large"}
    return {"kind": "serve", "games": _log(rng, 16, 256), "max_positions": _log(rng, 1000, 30000)}


# ---- inputs -------------------------------------------------------------------
def _job(row_seed, seed):
    """One job of the batched configuration with its states and its visible
    labels renumbered: (src, dst, label, p, q)."""
    src, dst, lab, p, q = synth.batched_lts(row_seed)
    rng = np.random.default_rng([row_seed, seed])
    n = int(max(src.max(), dst.max(), p, q)) + 1
    perm = rng.permutation(n).astype(np.uint32)
    lp = np.concatenate([[0], 1 + rng.permutation(int(lab.max()))]).astype(np.int32)
    return perm[src], perm[dst], lp[lab], int(perm[p]), int(perm[q])


def _near(positions):
    """The recorded job whose game is nearest to `positions`."""
    return _ROWS[min(int(np.searchsorted(_POS, positions)), len(_ROWS) - 1)]


def _spread(count, max_positions, seed, vary=False):
    """`count` recorded jobs evenly over all games of at most `max_positions`,
    in an order of the seed's; with `vary` other jobs of those sizes for every
    seed."""
    rng = np.random.default_rng(seed)
    m = int(np.searchsorted(_POS, max_positions, side="right"))
    at = (np.arange(count) + (rng.random(count) if vary else 0.5)) * (m / count)
    return [_ROWS[int(i)] for i in at[rng.permutation(count)]]


def _renumber(row, col, wt, att, seed):
    """The game with its positions in a random order (CSR arrays)."""
    n = len(att)
    new = np.random.default_rng(seed).permutation(n).astype(np.uint32)  # old -> new
    old = np.empty(n, dtype=np.int64)
    old[new] = np.arange(n)
    deg = np.diff(row.astype(np.int64))[old]
    row2 = np.zeros(n + 1, dtype=np.uint32)
    np.cumsum(deg, out=row2[1:])
    at = np.repeat(row[:-1].astype(np.int64)[old] - row2[:-1].astype(np.int64), deg)
    at += np.arange(len(at))
    return row2, new[col[at]], wt[at], att[old]


@functools.lru_cache(maxsize=1)
def _stress(n, m):
    return synth.scaled_stress_game(2, n, m)


def _system(row, seed):
    src, dst, lab, p, q = _job(row[1], seed)
    # a state without transitions may have got the largest number
    n = int(max(src.max(), dst.max(), p, q)) + 1
    return geq.TransitionSystem.from_arrays(src, dst, lab, n), p, q


def _graph(row, seed):
    lts, p, q = _system(row, seed)
    red, mapping = lts.bisimilar_minimize()
    return geq.GameBuild.compare(red, int(mapping[p]), int(mapping[q])).game


def _graphs(rows, seed):
    with ThreadPoolExecutor(max_workers=16) as ex:
        return list(ex.map(lambda r: _graph(r, seed), rows))


def _wide(elements, mx, n):
    """A bipartite game of a conf outside the one-word codecs: 60 % attackers,
    geometric out-degrees, updates 55 % zero, 30 % one decrement, 15 % one
    min-merge."""
    rng = np.random.default_rng(2)
    conf = geq.EnergyConf(elements, mx)
    att = (rng.random(n) < 0.6).astype(np.uint8)
    att[:2] = (1, 0)
    deg = rng.geometric(1.0 / 2.2, n).astype(np.int64) - (att == 0)
    row = np.zeros(n + 1, dtype=np.uint32)
    np.cumsum(deg, out=row[1:])
    m = int(row[-1])
    A, D = np.nonzero(att)[0].astype(np.uint32), np.nonzero(att == 0)[0].astype(np.uint32)
    from_att = np.repeat(att, deg).astype(bool)
    col = np.where(from_att, D[rng.integers(0, len(D), m)], A[rng.integers(0, len(A), m)])
    r = rng.random(m)
    pos = rng.integers(0, elements, m)
    code = np.where(r < 0.55, 0, 1)
    if elements > 1:
        tgt = rng.integers(0, elements - 1, m)
        tgt = tgt + (tgt >= pos)
        code = np.where(r < 0.85, code, tgt + 2)
    per = 32 // conf.update_bits()
    wt = np.zeros((m, conf.update_size()), dtype=np.uint32)
    wt[np.arange(m), pos // per] = code.astype(np.uint32) << (conf.update_bits() * (pos % per)).astype(np.uint32)
    return row, col, wt, att


_servers: dict = {}


def _server():
    """The process's server, as a program keeps one."""
    if "s" not in _servers:
        _servers["s"] = Server()
    return _servers["s"]


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "ctx": geq.default_context()}
    if kind == "game":
        st["graphs"] = [_graph(_near(case["positions"]), seed)]
    elif kind == "wide":
        arrays = _renumber(*_wide(case["elements"], case["max"], case["positions"]), seed)
        st["graphs"] = [geq.GameGraph.from_csr(*arrays, geq.EnergyConf(case["elements"], case["max"]))]
    elif kind in ("batch", "serve"):
        st["graphs"] = _graphs(_spread(case["games"], case["max_positions"], seed), seed)
    elif kind == "stress":
        arrays = _renumber(*_stress(case["positions"], case["edges"]), seed)
        st["graphs"] = [geq.GameGraph.from_csr(*arrays, geq.EnergyConf.STANDARD)]
    elif kind == "compare":
        st["jobs"] = [_system(r, seed) for r in _spread(case["jobs"], case["max_positions"], seed, vary=True)]
        st["together"] = case["together"]
    else:
        if case["family"] == "small":
            rng = np.random.default_rng(seed)
            n, m = case["states"], case["transitions"]
            arrays = (rng.integers(0, n, m), rng.integers(0, n, m), synth._labels(rng, m, 4, 0.2))
        else:
            arrays = synth.large_lts(seed, n=case["states"], m=case["transitions"])
        st["lts"] = geq.TransitionSystem.from_arrays(*arrays)
        st["relations"] = [geq.std_equivalences.get(x) for x in _RELATIONS]
    if kind in ("game", "wide", "batch"):
        st["views"] = geq.c_views(st["graphs"])
    if kind == "stress" or (kind == "batch" and case["resident"]):
        st["resident"] = geq.DeviceGames(st["graphs"], st["ctx"])
    if kind == "serve":
        st["server"] = _server()
    return st


# ---- one pass -----------------------------------------------------------------
class _Solution:
    """Frees a solution with the last array that views its memory."""

    def __init__(self, handle):
        self.handle = handle

    def __del__(self):
        lib.geq_solution_free(self.handle)


def _flat(sol):
    """A solution's offsets and energies: views of its memory."""
    owner = _Solution(sol)
    po, pd = C.POINTER(C.c_uint64)(), C.POINTER(C.c_uint32)()
    no, nw = C.c_uint64(), C.c_uint64()
    check(lib.geq_solution_flat(sol, C.byref(po), C.byref(no), C.byref(pd), C.byref(nw)))
    out = []
    for ptr, n, ctype, dtype in ((po, no.value, C.c_uint64, np.uint64), (pd, nw.value, C.c_uint32, np.uint32)):
        if n == 0:
            out.append(np.zeros(0, dtype))
            continue
        buf = (ctype * n).from_address(C.cast(ptr, C.c_void_p).value)
        buf._owner = owner
        out.append(np.frombuffer(buf, dtype=dtype))
    return out


def run(state):
    kind = state["kind"]
    if "resident" in state:
        games = state["resident"]
        games.solve()
        sol = C.c_void_p()
        check(lib.geq_device_games_download(games.ctx.h, games.h, C.byref(sol)))
        return _flat(sol)
    if kind in ("game", "wide", "batch"):
        sol = C.c_void_p()
        check(lib.geq_energy_game_run_batch(state["ctx"].h, len(state["graphs"]), state["views"], None, None, None,
                                            C.byref(sol)))
        return _flat(sol)
    if kind == "serve":
        server = state["server"]
        tickets = [server.submit(g) for g in state["graphs"]]
        got = [server.poll(t) for t in tickets]
        return [np.concatenate([x[0] for x in got]), np.concatenate([x[1] for x in got])]
    if kind == "compare":
        if state["together"]:
            lists = geq.compare_batch(state["jobs"], state["ctx"])
        else:
            lists = [lts.compare(p, q, state["ctx"]) for lts, p, q in state["jobs"]]
        table = np.zeros((len(lists), _WIDTH), dtype=np.uint32)
        for k, x in enumerate(lists):
            table[k, :len(x)] = x.array[:, 0]
        return [np.array([len(x) for x in lists]), table]
    eq = state["lts"].equivalences(state["ctx"])
    return [eq.relation(x).classes for x in state["relations"]]


# ---- what a pass cannot do without ---------------------------------------------
def _game_bytes(n, m):
    # CSR rows, successors, updates and attacker flags in; offsets and (about
    # two per position) energies out
    return 4 * (n + 1) + 8 * m + n + 8 * (n + 1) + 8 * n


def work(case):
    """Bytes that have to be read and written once; the path is integer work
    without floating-point operations."""
    kind = case["kind"]
    if kind == "game":
        n, _, m = _near(case["positions"])
        b = _game_bytes(n, m)
    elif kind in ("batch", "serve"):
        m = int(np.searchsorted(_POS, case["max_positions"], side="right"))
        b = case["games"] * _game_bytes(_POS[:m].mean(), _EDGES[:m].mean())
    elif kind == "stress":
        b = _game_bytes(case["positions"], case["edges"])
    elif kind == "wide":
        conf = geq.EnergyConf(case["elements"], case["max"])
        n, m = case["positions"], 1.8 * case["positions"]
        b = 13 * n + m * 4 * (1 + conf.update_size()) + 8 * n * conf.energy_size()
    elif kind == "compare":
        # a system (about 900 states and 2,900 transitions on average) in, a list of energies out
        b = case["jobs"] * (900 * 4 + 2900 * 8 + 16)
    else:
        # the system in, the lists of the ordered pairs of states with equal enabled labels (about 1 in 16)
        b = 4 * case["states"] + 8 * case["transitions"] + 8 * case["states"] ** 2 / 16
    return {"bytes": float(b), "flops": 0.0}


def exact(case, seed):
    """Every output is whole numbers: packed energies, offsets and class ids."""
    return None
