"""Multi-word solver: attackers whose successors only offer what they hold
already stay unchanged -- their lists are not written again and their
predecessors not visited.  Whether a kept energy is an own one is recorded by
one lane and read by another, so the lists span one to eight chunks of 32."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("conf", [(1, 0xFFFFFFFF), (2, 65535), (3, 1000), (4, 0xFFFFFFFF)])
@pytest.mark.parametrize("members", [1, 31, 32, 33, 64, 200, 256])
@pytest.mark.parametrize("n_chains", [40, 3000])
def test_unchanged_attackers(conf, members, n_chains):
    """Per chain: 3 (attacker, to reach) <- 2 (defender) <- 1 (attacker with
    the same list) <- 0 (defender).  Round 1 gives 2 the list of 3, round 2
    finds 1 unchanged: 0 is never visited."""
    import gpuequiv_b200 as geq
    from gpuequiv_b200._lib import check, geq_energy_lists, geq_solve_stats, lib
    el, mx = conf
    if el == 1:
        members = 1
    c = geq.EnergyConf(el, mx)
    v = np.zeros((members, el), np.uint64)
    if el > 1:
        v[:, 0] = np.arange(members)
        v[:, 1] = members - np.arange(members)
    per = 32 // c.energy_bits()
    one = np.zeros((members, c.energy_size()), np.uint32)
    for i in range(el):
        one[:, i // per] |= (v[:, i] << np.uint64(c.energy_bits() * (i % per))).astype(np.uint32)
    base = 4 * np.arange(n_chains, dtype=np.uint32)
    n = 4 * n_chains
    row = np.append((3 * np.arange(n_chains)[:, None] + np.array([0, 1, 2, 3])).reshape(-1), 3 * n_chains)
    col = (base[:, None] + np.array([1, 2, 3], np.uint32)).reshape(-1)
    wt = np.zeros((3 * n_chains, c.update_size()), np.uint32)
    att = np.tile(np.array([0, 1, 0, 1], np.uint8), n_chains)
    counts = np.tile(np.array([0, members, 0, members], np.uint64), n_chains)
    offs = np.zeros(n + 1, np.uint64)
    np.cumsum(counts, out=offs[1:])
    data = np.ascontiguousarray(np.tile(one, (2 * n_chains, 1)).reshape(-1))
    reach = np.ascontiguousarray(base + 3)
    ctx = geq.Context(0)
    g = geq.GameGraph.from_csr(row.astype(np.uint32), col, wt, att, c)
    view = g.c_view()
    init = geq_energy_lists(n, c.energy_size(), offs.ctypes.data_as(C.POINTER(C.c_uint64)),
                            data.ctypes.data_as(C.POINTER(C.c_uint32)))
    sol, st, out = C.c_void_p(), geq_solve_stats(), geq_energy_lists()
    check(lib.geq_energy_game_run(ctx.h, C.byref(view), C.byref(init), reach.ctypes.data_as(C.POINTER(C.c_uint32)),
                                  n_chains, C.byref(sol)))
    lib.geq_solution_stats(sol, C.byref(st))
    check(lib.geq_solution_lists(sol, 0, C.byref(out)))
    lens = np.diff(np.ctypeslib.as_array(out.offsets, shape=(n + 1,)).astype(np.int64)).reshape(-1, 4)
    lib.geq_solution_free(sol)
    ctx.close()
    # (energies of one 32-bit or two 16-bit fields are one-word confs: the same counts hold there)
    assert (st.rounds, st.positions_computed) == (2, 2 * n_chains)
    assert (lens == [0, members, members, members]).all()
