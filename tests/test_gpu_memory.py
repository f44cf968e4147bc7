"""Device memory: the budget a graph is created with, allocations that fail,
and buffers kept between calls. Failures are made by BF_TEST_FAIL_ALLOC (the
named allocation reports that the device's memory has run out)."""
import contextlib
import os

import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu
INF = 0xFFFFFFFF


@contextlib.contextmanager
def _env(name, value):
    os.environ[name] = value
    try:
        yield
    finally:
        del os.environ[name]


def _fails(what, call):
    import bfphast
    with _env("BF_TEST_FAIL_ALLOC", what), pytest.raises(bfphast.BfError) as e:
        call()
    assert e.value.status == bfphast.BF_ERR_OOM


def _without_panels(cch, **kw):
    import bfphast
    with _env("BF_TEST_FAIL_ALLOC", "panels"):
        return bfphast.Graph.from_cch(cch, **kw)


def test_isochrones_of_a_budget_at_one_tile(built):
    """Budgets around what a tile of 64 lanes and its scratch take: each is
    served, by the tile or by items."""
    import bfphast
    from test_gpu_panels import _band, _cch
    n, count = 180, 5
    cch = _cch(n, _band(n, 1), 3, 1, 60, 0.2)  # (its items take less than a tile)
    c = orc.Cch.from_dict(cch)
    org = np.arange(0, count * 30, 30, dtype=np.uint32)
    thr = np.full(count, 300, np.uint32)
    want, _ = c.isochrone_bitsets(org, thr)
    own = _without_panels(cch).info()["device_bytes"]
    tile = own + 128 * n + 2 * 4 * n + 4096 + 32 + 12 * count
    for budget in [tile + k for k in range(-4, 400, 4)] + [1 << 20, 4 << 20]:
        g = bfphast.Graph.from_cch(cch, hbm_budget=budget)
        assert np.array_equal(g.isochrone_bitsets(org, thr)[0], want), budget - tile


def test_graph_without_host_memory_for_panels(built, grid100):
    """Building the tiles runs out of host memory on worker threads: the graph is
    served without panels."""
    import bfphast
    _, cch = grid100
    with _env("BF_TEST_FAIL_ALLOC", "panel_tiles"):
        g = bfphast.Graph.from_cch(cch)
    assert g.info()["device_bytes"] == _without_panels(cch).info()["device_bytes"]
    src, tgt = (np.arange(k, cch["n"], 900, dtype=np.uint32) for k in (1, 5))
    assert np.array_equal(g.matrix(src, tgt), orc.Cch.from_dict(cch).matrix(src, tgt)[0])


def test_customization_without_room_for_panels(built):
    import bfphast
    from test_gpu_cch_panels import CASES, _topo
    _, n, pairs = CASES["tree"]
    rng = np.random.default_rng(1)
    t = _topo(n, pairs, rng, 0.3)
    with _env("BF_TEST_FAIL_ALLOC", "cch_panels"):
        g = bfphast.Cch.from_oracle_topo(t)
    up, dn = (rng.integers(0, 1000, len(x)).astype(np.uint32) for x in (t.up_mid, t.down_mid))
    got, want = g.relax(up, dn, t.up_mid, t.down_mid), t.relax(up, dn)[:4]
    assert all(np.array_equal(a, b) for a, b in zip(got, want))


def test_schedule_allocation_that_fails_is_given_back(built, country_small):
    import bfphast
    _, cch = country_small
    rng = np.random.default_rng(1)
    src, tgt = (rng.integers(0, cch["n"], k).astype(np.uint32) for k in (20, 300))
    g, h = bfphast.Graph.from_cch(cch), bfphast.Graph.from_cch(cch)
    for _ in range(2):
        _fails("panel_schedule", lambda: g.matrix(src, tgt))
    assert np.array_equal(g.matrix(src, tgt), h.matrix(src, tgt))
    assert g.info()["device_bytes"] == h.info()["device_bytes"]


def test_plain_slabs_are_allocated_all_or_none(built, grid100):
    """A call after one whose seed slab could not be allocated starts over."""
    import bfphast
    _, cch = grid100
    g = bfphast.Graph.from_cch(cch)
    g.set_engine(bfphast.ENGINE_PLAIN)
    src, tgt = (np.arange(k, cch["n"], 900, dtype=np.uint32) for k in (1, 5))
    for _ in range(2):
        _fails("plain_seeds", lambda: g.matrix(src, tgt))
    assert np.array_equal(g.matrix(src, tgt), orc.Cch.from_dict(cch).matrix(src, tgt)[0])


def _runs_graph(n, run=20):
    """n ranks in runs of 20, each joined to the next three of its run."""
    u = np.arange(n, dtype=np.int64)
    up = np.concatenate([np.stack([v := u[(u % run) < run - k], v + k], 1) for k in (1, 2, 3)])
    up = up[np.lexsort((up[:, 1], up[:, 0]))]
    w = np.random.default_rng(2).integers(1, 100, (2, len(up))).astype(np.uint32)
    o = np.lexsort((up[:, 0], up[:, 1]))
    off = np.zeros((2, n + 1), np.uint64)
    off[0, 1:] = np.cumsum(np.bincount(up[:, 0], minlength=n))
    off[1, 1:] = np.cumsum(np.bincount(up[:, 1], minlength=n))
    return dict(n=n, up_off=off[0], up_tgt=up[:, 1].astype(np.uint32), up_w=w[0],
                down_off=off[1], down_tgt=up[o, 0].astype(np.uint32), down_w=w[1][o])


def test_failed_call_keeps_no_large_buffer(built):
    """A call's buffer above the kept size is given back when the call fails too."""
    import torch

    import bfphast
    cch = _runs_graph(600_000)
    g = bfphast.Graph.from_cch(cch)
    src = np.arange(0, 128 * 4000, 4000, dtype=np.uint32)  # 307 MB of distances
    one = g.query_batch(src[:1])
    free = torch.cuda.mem_get_info()[0]
    with _env("BF_TEST_WITHHOLD_ARRIVAL", "1"), pytest.raises(bfphast.BfError) as e:
        g.query_batch(src)
    assert e.value.status == bfphast.BF_ERR_TIMEOUT
    assert free - torch.cuda.mem_get_info()[0] < 4 * cch["n"] * len(src) // 2
    assert np.array_equal(g.query_batch(src[:1]), one)


def _served(make, want):
    """Whether a graph's calls are served; a budget too small is BF_ERR_OOM."""
    import bfphast
    try:
        g = make()
        for call, w in want:
            assert np.array_equal(call(g), w)
    except bfphast.BfError as e:
        assert e.status == bfphast.BF_ERR_OOM
        return None
    return g


@pytest.mark.parametrize("two", [False, True])
def test_budget_covers_panels(built, country_small, two):
    """What a graph with a budget holds stays within it, its panels too, and no
    budget that serves a call without panels is too small with them."""
    import bfphast
    _, cch = country_small
    n = cch["n"]
    c = orc.Cch.from_dict(cch)
    rng = np.random.default_rng(2)
    src = rng.integers(0, n, 40).astype(np.uint32)
    tgt = rng.choice(n, 500, replace=False).astype(np.uint32)
    thr = np.full(3, 9000, np.uint32)
    kw = {}
    want = [(lambda g: g.matrix(src, tgt), c.matrix(src, tgt)[0]),
            (lambda g: g.isochrone_bitsets(src[:3], thr)[0], c.isochrone_bitsets(src[:3], thr)[0])]
    if two:
        ln = [np.where(cch[k] == INF, cch[k], cch[k] // 2 + 1) for k in ("up_w", "down_w")]
        kw = dict(up_len=ln[0], down_len=ln[1])
        sets = [[[(int(r), 1, 2)] for r in x[:40]] for x in (src, tgt)]
        want.append((lambda g: g.matrix_seeded_2ch(*sets)[1],
                     orc.table_phast_lopsided_2ch(c, *sets, INF, *ln)[1]))
    with_panels = 0
    last = False
    for mb in list(range(12, 60, 2)) + list(range(64, 400, 16)):
        budget = mb << 20
        g = _served(lambda: bfphast.Graph.from_cch(cch, hbm_budget=budget, **kw), want)
        h = _served(lambda: _without_panels(cch, hbm_budget=budget, **kw), want)
        assert (g is not None) == (h is not None), mb
        assert g is not None or not last, mb
        last = g is not None
        if g is None:
            continue
        assert g.info()["device_bytes"] <= budget, mb
        fresh = bfphast.Graph.from_cch(cch, hbm_budget=budget, **kw).info()["device_bytes"]
        with_panels += fresh > _without_panels(cch, hbm_budget=budget, **kw).info()["device_bytes"]
    assert last and with_panels


def test_serving_slot_budgets(built, country_small):
    """Slots whose budget holds 32 lanes of the rows that reach a target but not
    of the targets' ancestors sweep items; tables and isochrones, budgets from too
    small to ample."""
    import time

    import bfphast
    _, cch = country_small
    n = cch["n"]
    c = orc.Cch.from_dict(cch)
    rng = np.random.default_rng(2)
    src = rng.integers(0, n, 40).astype(np.uint32)
    tgt = rng.choice(n, 500, replace=False).astype(np.uint32)
    want, _ = c.matrix(src, tgt)
    want_bits, _ = c.isochrone_bitsets(src[:1], np.array([9000], np.uint32))
    g = bfphast.Graph.from_cch(cch)
    served = []
    for kb in list(range(600, 3000, 100)) + [8000, 20000, 64000]:
        srv = bfphast.Server(g, hbm_budget=2 * kb << 10, slots=1)
        t, out = srv.submit_matrix(src, tgt)
        ti, bits = srv.submit_isochrone(int(src[0]), 9000)
        done, t0 = {}, time.time()
        while len(done) < 2 and time.time() - t0 < 60:
            done.update({x["ticket"]: x["status"] for x in srv.poll(wait_ms=200)})
        srv.close()
        assert set(done.values()) <= {bfphast.BF_OK, bfphast.BF_ERR_OOM}, kb
        if done[t] == bfphast.BF_OK:
            assert np.array_equal(out, want), kb
        if done[ti] == bfphast.BF_OK:
            assert np.array_equal(bits, want_bits[0]), kb
        served.append((done[t] == bfphast.BF_OK, done[ti] == bfphast.BF_OK))
    for k in (0, 1):  # from some budget on
        s = [x[k] for x in served]
        assert s == sorted(s) and s[-1] and not s[0], (k, s)
