"""Games of very many rounds: the time limit between steps holds for lone games
of every size above 4,096 positions, and in the server they do not hold up
other requests."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def chain(geq, n):
    row = np.minimum(np.arange(n + 1), n - 1).astype(np.uint32)
    att = (np.arange(n) % 2 != (n - 1) % 2).astype(np.uint8)  # the last position is a defender
    return geq.GameGraph.from_csr(row, np.arange(1, n, dtype=np.uint32), np.zeros(n - 1, np.uint32), att,
                                  geq.EnergyConf.STANDARD)


@pytest.mark.parametrize("n", [4097, 4098, 20000, 32768, 32769])
def test_time_limit(monkeypatch, n):
    import gpuequiv_b200 as geq
    ctx = geq.Context(0)
    g = chain(geq, n)
    offs, data, stats = geq.run_batch_raw([g], ctx)
    assert stats["rounds"] >= n - 1
    assert np.array_equal(offs[0], np.arange(n + 1)) and not data[0].any()
    if n > 5000:  # (up to 4,096 rounds in one launch)
        monkeypatch.setenv("GEQ_SOLVE_TIMEOUT_S", "0.0001")
        with pytest.raises(geq.GeqError, match="no fixpoint"):
            geq.run_batch_raw([g], ctx)
        monkeypatch.delenv("GEQ_SOLVE_TIMEOUT_S")
        offs, data, _ = geq.run_batch_raw([g], ctx)  # the context goes on
        assert np.array_equal(offs[0], np.arange(n + 1)) and not data[0].any()
    ctx.close()


def test_server_short_beside_long():
    """One pipeline: a chain of 32,000 rounds (some 0.2 s) and then short games,
    lone requests all; the short ones are answered while the chain is solved."""
    import gpuequiv_b200 as geq
    from gpuequiv_b200.serving import Server
    ctx = geq.Context(0)
    long, short = chain(geq, 32000), chain(geq, 20)
    with Server(ctx, n_pipelines=1) as srv:
        for g in (short, long):  # everything allocated and loaded
            srv.poll(srv.submit(g))
        t = srv.submit(long)
        assert srv.poll(t, 5) is None  # taken by the pipeline
        early = 0
        for _ in range(5):
            got = srv.poll(srv.submit(short))
            assert np.array_equal(got[0], np.arange(21))
            early += srv.stats()["running"] >= 1  # the chain
        assert early == 5
        got = srv.poll(t)
        assert np.array_equal(got[0], np.arange(32001)) and not got[1].any()
    ctx.close()


@pytest.mark.parametrize("n", [2000, 50000])
def test_levels_per_launch(n):
    """GameBuild of two chains that differ at their ends: a level per position
    and more, at most 4,096 levels a launch."""
    import gpuequiv_b200 as geq
    ctx = geq.Context(0)
    s = np.arange(n - 1)
    src, dst = np.concatenate([s, s + n]), np.concatenate([s + 1, s + 1 + n])
    label = np.concatenate([np.ones(n - 1), np.ones(n - 1)]).astype(np.int32)
    label[-1] = 2
    lts = geq.TransitionSystem.from_arrays(src.astype(np.uint32), dst.astype(np.uint32), label, 2 * n)
    geq.GameBatch([(lts, 0, n)], ctx)  # the next build starts with buffers of its size
    b = geq.GameBatch([(lts, 0, n)], ctx)
    exp = geq.GameBuild.compare(lts, 0, n).game
    got = b.graph(0)
    for f in ("row_offsets", "column_indices", "attacker_pos"):
        assert np.array_equal(getattr(got, f), getattr(exp, f)), f
    info = b.stats
    assert info["levels"] >= n
    assert info["kernel_launches"] >= 1 + -(-info["levels"] // 4096)  # and the assembly's
    ctx.close()
