"""Graphs with no edges, or with edges in one direction only, through every entry
point, against the oracle: schedules without work items, waves without levels."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu
INF = 0xFFFFFFFF


def _cch(n, up, down):
    """A chain with the chosen directions; the others hold INF weights."""
    off = np.minimum(np.arange(n + 1), n - 1).astype(np.uint64)
    doff = np.concatenate([[0], np.arange(n)]).astype(np.uint64)
    w = np.arange(1, n, dtype=np.uint32)
    gone = np.full(n - 1, INF, np.uint32)
    return dict(n=n, up_off=off, up_tgt=np.arange(1, n, dtype=np.uint32), up_w=w if up else gone,
                down_off=doff, down_tgt=np.arange(0, n - 1, dtype=np.uint32),
                down_w=w if down else gone)


@pytest.mark.parametrize("n", [1, 7, 40])
@pytest.mark.parametrize("up", [0, 1])
@pytest.mark.parametrize("down", [0, 1])
@pytest.mark.parametrize("dev", [1, 0])
def test_every_call(built, n, up, down, dev):
    import bfphast
    cch = _cch(n, up, down)
    c = orc.Cch.from_dict(cch)
    g = bfphast.Graph.from_cch(cch)
    g.set_tune(device_schedule=dev)
    every = np.arange(n, dtype=np.uint32)
    want, _ = c.matrix(every, every)
    for eng in (bfphast.ENGINE_PLAIN, bfphast.ENGINE_BATCHED):
        g.set_engine(eng)
        assert np.array_equal(g.matrix(every, every), want), eng
    assert np.array_equal(g.query_batch(every), want)
    for top in (3, 0xFFFE, 0xFFFF, INF):
        for persist in (1, 3):
            g.set_tune(device_schedule=dev, persistent_sweep=persist)
            thr = np.full(n, top, np.uint32)
            bits, counts = g.isochrone_bitsets(every, thr)
            wb, wc = c.isochrone_bitsets(every, thr)
            assert np.array_equal(bits, wb) and np.array_equal(counts, wc), (top, persist)
    sets = [[(int(r), 1)] for r in every]
    assert np.array_equal(g.matrix_seeded(sets, sets), orc.table_phast_lopsided(c, sets, sets, INF)[0])
    got, ref = g.phast_bounded_seeded([(0, 0)], 9), c.bounded_seeded([(0, 0)], 9)
    assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])
