"""Graphs whose panels do not fit the device: every call runs over single rows
(work items, launches a level, the persistent sweep of rows), against the
oracle, tolerance 0. Most of these forms serve other cases too (host-built
schedules, thresholds beyond 16 bits, trees too deep for shared memory); here
they are the device-built schedule's peeling and its deadline, the plain
engine's persistent sweep and its deadline, the upward pass by runs, and the
isochrone waves by items.

The panels are left out by BF_TEST_FAIL_ALLOC=panels: their allocation fails as
on a device without room for them."""
import contextlib
import os

import numpy as np
import pytest

from oracle import oracle as orc
from test_gpu_deep import _zigzag

pytestmark = pytest.mark.gpu
INF = 0xFFFFFFFF


@contextlib.contextmanager
def _env(name, value):
    os.environ[name] = value
    try:
        yield
    finally:
        del os.environ[name]


def _without_panels(cch, **kw):
    import bfphast
    with _env("BF_TEST_FAIL_ALLOC", "panels"):
        g = bfphast.Graph.from_cch(cch, **kw)
    h = bfphast.Graph.from_cch(cch, **kw)
    assert g.info()["device_bytes"] < h.info()["device_bytes"]  # (the hook took effect)
    h.close()
    return g


def _timeout(call):
    import bfphast
    with _env("BF_TEST_WITHHOLD_ARRIVAL", "1"), pytest.raises(bfphast.BfError) as e:
        call()
    assert e.value.status == bfphast.BF_ERR_TIMEOUT


@pytest.fixture(params=["grid100", "country_small"])
def cch(request):
    return request.getfixturevalue(request.param)[1]


def test_device_and_host_schedules_agree(built, cch):
    n = cch["n"]
    c = orc.Cch.from_dict(cch)
    g = _without_panels(cch)
    rng = np.random.default_rng(21)
    src = rng.choice(n, 40, replace=False).astype(np.uint32)
    full = np.stack([c.phast_query(s) for s in src])
    cases = [rng.choice(n, 300), np.arange(n - 40, n), np.arange(0, 40), [7], rng.choice(n, 5000)]
    for tgt in cases:
        tgt = np.asarray(tgt, np.uint32)
        got = {}
        for dev in (1, 0):
            g.set_tune(device_schedule=dev)
            m, st = g.matrix(src, tgt, stats=True)
            assert np.array_equal(m, full[:, tgt]), (dev, len(tgt))
            levels = [x.tolist() for x in g.schedule_levels()]
            got[dev] = (st["swept_nodes"], st["swept_edges"], levels)
            m = g.matrix(src, tgt, threshold=1800)
            assert np.array_equal(m, np.where(full[:, tgt] <= 1800, full[:, tgt], INF)), dev
        assert got[0] == got[1], len(tgt)


def test_peeling_deadline(built, cch):
    """Rows are only taken off a schedule when nothing reads them: what a
    timed-out peeling leaves is a correct superset, and the call fails."""
    n = cch["n"]
    c = orc.Cch.from_dict(cch)
    g = _without_panels(cch)
    src = np.array([3, 1000, 30000, 17], np.uint32)
    for first in (5, 11):
        tgt = np.arange(first, n, 97, dtype=np.uint32)
        _timeout(lambda: g.matrix(src, tgt))
        want, _ = c.matrix(src, tgt)
        assert np.array_equal(g.matrix(src, tgt), want)


def test_plain_persistent_sweep_of_rows(built, cch):
    import bfphast
    n = cch["n"]
    c = orc.Cch.from_dict(cch)
    g = _without_panels(cch)
    g.set_engine(bfphast.ENGINE_PLAIN)
    rng = np.random.default_rng(4)
    src = rng.choice(n, 70, replace=False).astype(np.uint32)
    tgt = rng.choice(n, 500, replace=False).astype(np.uint32)
    want, _ = c.matrix(src, tgt)
    _timeout(lambda: g.matrix(src, tgt))
    for persist in (1, 0):
        g.set_tune(persistent_sweep=persist)
        got, st = g.matrix(src, tgt, stats=True)
        assert np.array_equal(got, want), persist
        if persist:
            assert st["kernel_launches"] == 3 * 3 + 1
        m = g.matrix(src, tgt, threshold=2000)
        assert np.array_equal(m, np.where(want <= 2000, want, INF)), persist
    assert np.array_equal(g.query_batch(src[:3]), np.stack([c.phast_query(s) for s in src[:3]]))


@pytest.mark.parametrize("count", [1, 40, 200, 300])
def test_isochrones_by_items(built, cch, count):
    import workload
    c = orc.Cch.from_dict(cch)
    g = _without_panels(cch)
    origins, thr = workload.isochrone_workload(cch["n"], count, seed=count)
    bits, counts = g.isochrone_bitsets(origins, thr)
    want_bits, want_counts = c.isochrone_bitsets(origins, thr)
    assert np.array_equal(bits, want_bits) and np.array_equal(counts, want_counts)
    sets = g.isochrone_settled(origins[:9], thr[:9])
    for i, (rk, ds) in enumerate(sets):
        wr, wd = c.bounded_seeded([(int(origins[i]), 0)], int(thr[i]))
        assert np.array_equal(rk, wr) and np.array_equal(ds, wd), i


def test_seeded_tables_by_items(built, cch):
    n = cch["n"]
    ln = [np.where(cch[k] == INF, cch[k], cch[k] // 2 + 1) for k in ("up_w", "down_w")]
    c = orc.Cch.from_dict(cch)
    g = _without_panels(cch, up_len=ln[0], down_len=ln[1])
    rng = np.random.default_rng(6)
    sets = [[[(int(rng.integers(0, n)), int(rng.integers(0, 90)), int(rng.integers(0, 500)))
              for _ in range(int(rng.integers(1, 4)))] for _ in range(m)] for m in (35, 50)]
    one = [[[s[:2] for s in x] for x in side] for side in sets]
    assert np.array_equal(g.matrix_seeded(*one), orc.table_phast_lopsided(c, *one, INF)[0])
    got = g.matrix_seeded_2ch(*sets)
    want = orc.table_phast_lopsided_2ch(c, *sets, INF, ln[0], ln[1])
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


@pytest.mark.parametrize("n", [60, 62, 64, 66, 400])
def test_upward_by_runs_and_by_nodes(built, n):
    """Ancestor paths of up to 32 runs (28 to 33 here) are walked by runs, longer
    ones by nodes: tables of both engines, bounds a lane, seed costs."""
    import bfphast
    cch = _zigzag(n)
    c = orc.Cch.from_dict(cch)
    g = _without_panels(cch)
    every = np.arange(n, dtype=np.uint32)
    want, _ = c.matrix(every, every)
    for eng in (bfphast.ENGINE_BATCHED, bfphast.ENGINE_PLAIN):
        g.set_engine(eng)
        for overlap in (1, 0):
            g.set_tune(overlap_upward=overlap)
            assert np.array_equal(g.matrix(every, every), want), (eng, overlap)
            assert np.array_equal(g.matrix(every, every, threshold=150),
                                  np.where(want <= 150, want, INF)), (eng, overlap)
    thr = (every * 37) % np.uint32(500)
    bits, counts = g.isochrone_bitsets(every, thr)
    want_bits, want_counts = c.isochrone_bitsets(every, thr)
    assert np.array_equal(bits, want_bits) and np.array_equal(counts, want_counts)
    for seeds in ([(0, 3), (n // 2, 0)], [(n - 1, 1)]):
        got, want1 = g.phast_bounded_seeded(seeds, 300), c.bounded_seeded(seeds, 300)
        assert np.array_equal(got[0], want1[0]) and np.array_equal(got[1], want1[1])
