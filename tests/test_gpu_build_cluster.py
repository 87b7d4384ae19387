"""GameBuild levels with small frontiers inside one launch: batches whose start
positions, frontiers and states sit around the lines of that path (1 job, the
4,096-position line of the start level and of a level, jobs with more states
than the per-warp bitmap), against the host builder, with and without it
(GEQ_TUNE_NO_GRAPH runs every level as plain launches)."""
from __future__ import annotations

import numpy as np
import pytest

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


def system(geq, seed, n, density, labels):
    rng = np.random.default_rng(seed)
    m = max(1, int(n * density))
    lab = rng.integers(0, labels, m)
    return geq.TransitionSystem.from_arrays(rng.integers(0, n, m), rng.integers(0, n, m), lab, n)


def same(got, exp):
    for f in ("row_offsets", "column_indices", "attacker_pos"):
        assert np.array_equal(getattr(got, f), getattr(exp, f)), f
    assert np.array_equal(got.weights.array, exp.weights.array)


@pytest.mark.parametrize("jobs", [1, 2, 33, 4095, 4096, 4097])
def test_compare_batches_around_the_start_line(geq, ctx, jobs):
    systems = [system(geq, s, 8 + 3 * s, 1.6, 3) for s in range(7)]
    work = [(systems[j % 7], j % 8, (j + 1 + j // 8) % 8) for j in range(jobs)]
    b = geq.GameBatch(work, ctx)
    for j in sorted({0, 1, jobs // 2, jobs - 1} & set(range(jobs))):
        lts, p, q = work[j]
        same(b.graph(j), geq.GameBuild.compare(lts, p, q).game)


@pytest.mark.parametrize("n,density,labels", [(2, 1.0, 1), (40, 3.0, 4), (130, 2.0, 5), (700, 1.2, 9),
                                              (40_000, 1.05, 30)])
def test_levels_of_one_system(geq, ctx, n, density, labels):
    """From a few positions a level to several thousand (both ways over the
    line), and a system with more states than the warp bitmap holds."""
    lts = system(geq, 5, n, density, labels)
    if n <= 700:
        b = geq.GameBatch.compare_all([lts], ctx)
        exp, _ = geq.GameBuild.compare_all(lts)
    else:
        b = geq.GameBatch([(lts, 3, 11)], ctx)
        exp = geq.GameBuild.compare(lts, 3, 11)
    same(b.graph(0), exp.game)


@pytest.mark.parametrize("bound", [1, 50, 5000])
def test_position_bound(geq, ctx, bound):
    lts = system(geq, 9, 60, 2.4, 4)
    full = geq.GameBuild.compare(lts, 1, 2).game
    b = geq.GameBatch([(lts, 1, 2), (lts, 1, 1)], ctx, max_positions=bound)
    if full.n_vertices() > bound:
        with pytest.raises(geq.GeqError):
            b.graph(0)
    else:
        same(b.graph(0), full)
