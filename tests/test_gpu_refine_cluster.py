"""Minimisation of small batches in one launch against the host's: states and
jobs around its lines (16,384 states), systems that need many iterations
(chains), single states; and compare() of pairs
that fall into one class beside pairs that do not."""
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


def chain(geq, n):
    return geq.TransitionSystem.from_arrays(np.arange(n - 1), np.arange(1, n), np.ones(n - 1, np.int32), n)


def random_system(geq, seed, n, density=2.0, labels=2):
    rng = np.random.default_rng(seed)
    m = int(n * density)
    return geq.TransitionSystem.from_arrays(rng.integers(0, n, m), rng.integers(0, n, m), rng.integers(0, labels, m), n)


@pytest.mark.parametrize("n", [1, 2, 33, 1000, 16383, 16384, 16385])
def test_sizes(geq, ctx, n):
    systems = [random_system(geq, n, n, 1.3), chain(geq, 2)]
    for (part, cnt), lts in zip(geq.signature_refinement_batch(systems, ctx), systems):
        exp, m = lts.signature_refinement()
        assert cnt == m and np.array_equal(part, exp)


@pytest.mark.parametrize("n", [3, 64, 300])
def test_many_iterations(geq, ctx, n):
    systems = [chain(geq, n), random_system(geq, 3, n), chain(geq, 5)]
    for (part, cnt), lts in zip(geq.signature_refinement_batch(systems, ctx), systems):
        exp, m = lts.signature_refinement()
        assert cnt == m and np.array_equal(part, exp)


@pytest.mark.parametrize("jobs", [1, 5, 700])
def test_compare_with_bisimilar_pairs(geq, ctx, jobs):
    lts = geq.TransitionSystem([(0, 1, 1), (1, 2, 2), (3, 4, 1), (4, 5, 2), (3, 6, 1), (7, 8, 1), (8, 9, 2)])
    pairs = [(0, 7), (0, 3), (3, 0), (2, 5), (1, 8)]
    work = [(lts, *pairs[k % 5]) for k in range(jobs)]
    exp = {pq: sorted(lts.compare_unminimized(*pq, ctx).array[:, 0].tolist()) for pq in pairs if pq in ((0, 3), (3, 0))}
    for (_, p, q), got in zip(work, geq.compare_batch(work, ctx)):
        assert sorted(got.array[:, 0].tolist()) == exp.get((p, q), [])
