"""Device memory of the multi-word solver: a large scratch of the warps goes back
to the device after the solve."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

# a process of its own: GameBuild makes the device's pool keep its blocks
CODE = """
import ctypes as C, itertools
import numpy as np, torch
import gpuequiv_b200 as geq
from gpuequiv_b200._lib import check, geq_energy_lists, lib
ctx = geq.Context(0)
c = geq.EnergyConf(80, 1)  # three words an energy, a bit a field
triples = np.array(list(itertools.islice(itertools.combinations(range(80), 3), 0, 82160, 13))[:6000])
words = np.zeros((len(triples), 3), np.uint32)
for k in range(3):
    for w in range(3):
        at = triples[:, k] // 32 == w
        words[at, w] |= np.uint32(1) << (triples[at, k] % 32).astype(np.uint32)
def solve(members):  # 0 (attacker) -> 1 (defender) -> 2 (attacker with the list)
    g = geq.GameGraph.from_csr(np.array([0, 1, 2, 2], np.uint32), np.array([1, 2], np.uint32),
                               np.zeros((2, c.update_size()), np.uint32), np.array([1, 0, 1], np.uint8), c)
    view = g.c_view()
    offs, data = np.array([0, 0, 0, members], np.uint64), np.ascontiguousarray(words[:members].reshape(-1))
    init = geq_energy_lists(3, 3, offs.ctypes.data_as(C.POINTER(C.c_uint64)), data.ctypes.data_as(C.POINTER(C.c_uint32)))
    reach = np.array([2], np.uint32)
    sol, out = C.c_void_p(), geq_energy_lists()
    check(lib.geq_energy_game_run(ctx.h, C.byref(view), C.byref(init), reach.ctypes.data_as(C.POINTER(C.c_uint32)), 1,
                                  C.byref(sol)))
    check(lib.geq_solution_lists(sol, 0, C.byref(out)))
    assert [int(out.offsets[i]) for i in range(4)] == [0, members, 2 * members, 3 * members]
    lib.geq_solution_free(sol)
solve(10)
torch.cuda.synchronize()
before = torch.cuda.mem_get_info(0)[0]
solve(6000)  # outgrows the smallest scratch, then its eightfold is 1.2 GB
solve(10)
torch.cuda.synchronize()
print("kept", before - torch.cuda.mem_get_info(0)[0])
"""


def test_scratch_goes_back():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CODE], capture_output=True, text=True, cwd=root, timeout=300)
    assert r.returncode == 0, r.stderr
    kept = int(r.stdout.split("kept")[1])
    assert kept < 256 << 20, kept
