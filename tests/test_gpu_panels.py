"""Panel sweeps (up to 16 consecutive ranks of one run swept as a dense tile)
against the CPU oracle and the item sweep (tolerance 0: u32 min-plus), at the
edges of panels, of weight-tile strides, of staged source chunks and of lane
blocks, and with labels beyond the one-instruction relaxation's range."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu
INF = 0xFFFFFFFF


def _cch(n, up, seed, w_lo, w_hi, drop):
    """CCH from UP neighbour lists; every edge also goes DOWN with its own
    weight, each direction dropped (INF) with probability `drop`, except the
    steps r -> r + 1 that make the runs."""
    rng = np.random.default_rng(seed)
    src = np.array([u for u in range(n) for _ in up[u]], np.int64)
    tgt = np.array([v for u in range(n) for v in up[u]], np.int64)
    w = rng.integers(w_lo, w_hi, (2, len(src)), dtype=np.uint64)
    w[:, (rng.random(len(src)) < drop) & (tgt != src + 1)] = INF
    lone = rng.random((2, len(src))) < drop
    lone[:, tgt == src + 1] = False
    w[lone] = INF
    off = np.zeros((2, n + 1), np.uint64)
    off[0, 1:] = np.cumsum(np.bincount(src, minlength=n))
    off[1, 1:] = np.cumsum(np.bincount(tgt, minlength=n))
    o = np.lexsort((src, tgt))
    return dict(n=n, up_off=off[0], up_tgt=tgt.astype(np.uint32), up_w=w[0].astype(np.uint32),
                down_off=off[1], down_tgt=src[o].astype(np.uint32),
                down_w=w[1][o].astype(np.uint32))


def _band(n, width):
    """One run of n ranks, each joined to the next `width`."""
    return [list(range(u + 1, min(n, u + 1 + width))) for u in range(n)]


def _fan():
    """A run whose 16 rows pull from disjoint ancestors (its tile is split),
    under a run of 700 ranks."""
    up = [[u + 1] + list(range(16 + 40 * u, 56 + 40 * u)) for u in range(16)]
    up[15] = sorted(set(up[15]))
    return [sorted(set(x)) for x in up] + [
        list(range(u + 1, min(716, u + 4))) for u in range(16, 716)]


GRAPHS = {
    # run lengths at and beside the panel and stride edges
    **{"band%d" % n: (_band(n, n), 1, 60) for n in (1, 2, 3, 5, 9, 13, 16, 17, 33)},
    "sources300": (_band(330, 330), 1, 1000),  # over 256 sources above a panel
    "fan": (_fan(), 1, 500),
    # labels up to and past 2^31, and sums that saturate
    "long": (_band(40, 12), 1 << 26, 1 << 28),
    "saturating": (_band(40, 12), 1 << 29, 0xFFFFFFF0),
}


@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_panels_small_graphs(built, name):
    import bfphast
    up, lo, hi = GRAPHS[name]
    n = len(up)
    cch = _cch(n, up, 7, lo, hi, 0.2)
    c = orc.Cch.from_dict(cch)
    g, items = bfphast.Graph.from_cch(cch), bfphast.Graph.from_cch(cch)
    items.set_tune(device_schedule=0)
    rng = np.random.default_rng(n)
    for S, T in ((1, 1), (4, n), (33, 5), (65, n), (129, 3), (600, n)):
        src = rng.integers(0, n, S).astype(np.uint32)
        tgt = rng.integers(0, n, T).astype(np.uint32)
        want, _ = c.matrix(src, tgt)
        got, st = g.matrix(src, tgt, stats=True)
        assert np.array_equal(got, want), (S, T)
        ref, si = items.matrix(src, tgt, stats=True)
        assert np.array_equal(ref, want), (S, T)
        assert (st["swept_nodes"], st["swept_edges"]) == (si["swept_nodes"], si["swept_edges"])
        sets = [[(int(s), int(rng.integers(0, 1 << 31)))] for s in src[:9]]
        tsets = [[(int(t), 0)] for t in tgt[:9]]
        got = g.matrix_seeded(sets, tsets)  # seed costs past the short range
        assert np.array_equal(got, orc.table_phast_lopsided(c, sets, tsets, INF)[0]), (S, T)


@pytest.mark.parametrize("name", ["band2", "band16", "band17", "band33", "sources300", "fan"])
def test_upward_by_panels_with_thresholds(built, name):
    """The upward pass with a threshold per lane (16-bit lanes), with seed
    costs, and entering a run at every row of a panel."""
    import bfphast
    up, lo, hi = GRAPHS[name]
    n = len(up)
    cch = _cch(n, up, 7, lo, hi, 0.2)
    c = orc.Cch.from_dict(cch)
    g = bfphast.Graph.from_cch(cch)
    org = np.arange(n, dtype=np.uint32)
    thr = (np.arange(n, dtype=np.uint32) * 7) % np.uint32(3 * hi)
    bits, counts = g.isochrone_bitsets(org, thr)
    want_bits, want_counts = c.isochrone_bitsets(org, thr)
    assert np.array_equal(bits, want_bits) and np.array_equal(counts, want_counts)
    for o in sorted({0, n // 3, n // 2, n - 1}):
        for t in (0, hi, INF):
            seeds = [(o, 3), (n // 2, 0), (min(n - 1, o + 5), hi)]
            got, want = g.phast_bounded_seeded(seeds, t), c.bounded_seeded(seeds, t)
            assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1]), (o, t)


@pytest.mark.parametrize("S", [64, 68, 100, 128, 130, 512, 516, 1030])
def test_panels_wide_levels(built, grid100, S):
    """Every node a target: levels of thousands of panels, lane blocks of 512
    and what is left of them, every block size."""
    import bfphast
    _, cch = grid100
    n = cch["n"]
    g = bfphast.Graph.from_cch(cch)
    rng = np.random.default_rng(S)
    src = rng.integers(0, n, S).astype(np.uint32)
    tgt = np.arange(n, dtype=np.uint32)
    pick = rng.choice(S, 12, replace=False)
    c = orc.Cch.from_dict(cch)
    want = np.stack([c.phast_query(int(s)) for s in src[pick]])
    for tpb in (32, 64, 128, 256):
        g.set_tune(threads_per_block=tpb)
        assert np.array_equal(g.matrix(src, tgt)[pick], want), tpb


def test_panels_budget_falls_back_to_items(built, country_small):
    """A budget for 32 lanes of the rows that reach a target, but not of the
    targets' ancestors, is still served (by the item sweep)."""
    import bfphast
    _, cch = country_small
    n = cch["n"]
    c = orc.Cch.from_dict(cch)
    rng = np.random.default_rng(2)
    src = rng.integers(0, n, 40).astype(np.uint32)
    tgt = rng.choice(n, 500, replace=False).astype(np.uint32)
    want, _ = c.matrix(src, tgt)
    served = 0
    for mb in range(12, 60, 2):
        g = bfphast.Graph.from_cch(cch, hbm_budget=mb << 20)
        try:
            for _ in range(2):
                assert np.array_equal(g.matrix(src, tgt), want), mb
            served += 1
        except bfphast.BfError as e:
            assert e.status == bfphast.BF_ERR_OOM and not served, mb
        g.close()
    assert served


@pytest.mark.parametrize("count", [1, 63, 64, 65, 129, 2100])
@pytest.mark.parametrize("top", [300, 0x7FFE, 0x7FFF, 0xFFFE])
def test_isochrones_by_panels(built, count, top):
    """Lanes at the edges of tiles and waves, thresholds at the edges of the
    two 16-bit forms: bitsets, counts and settled lists."""
    import bfphast
    up, lo, hi = _band(180, 60), 1, max(2, top // 40)
    n = len(up)
    cch = _cch(n, up, 3, lo, hi, 0.2)
    c = orc.Cch.from_dict(cch)
    g = bfphast.Graph.from_cch(cch)
    g.set_tune(isochrone_lanes=0)
    rng = np.random.default_rng(count)
    org = rng.integers(0, n, count).astype(np.uint32)
    thr = rng.integers(0, top + 1, count).astype(np.uint32)
    thr[0] = top
    bits, counts = g.isochrone_bitsets(org, thr)
    want_bits, want_counts = c.isochrone_bitsets(org, thr)
    assert np.array_equal(bits, want_bits) and np.array_equal(counts, want_counts)
    sets = g.isochrone_settled(org, thr)
    for i in range(0, count, max(1, count // 9)):
        rk, ds = c.bounded_seeded([(int(org[i]), 0)], int(thr[i]))
        assert np.array_equal(sets[i][0], rk) and np.array_equal(sets[i][1], ds), i


def test_isochrones_panels_budget_falls_back(built, country_small):
    """A budget below one tile of 64 lanes is still served (by the item waves)."""
    import bfphast
    _, cch = country_small
    c = orc.Cch.from_dict(cch)
    org = np.array([5, 700, 33000], np.uint32)
    thr = np.array([3000, 36000, 6000], np.uint32)
    want_bits, want_counts = c.isochrone_bitsets(org, thr)
    served = 0
    for mb in range(20, 60, 2):
        g = bfphast.Graph.from_cch(cch, hbm_budget=mb << 20)
        try:
            bits, counts = g.isochrone_bitsets(org, thr)
            assert np.array_equal(bits, want_bits) and np.array_equal(counts, want_counts), mb
            served += 1
        except bfphast.BfError as e:
            assert e.status == bfphast.BF_ERR_OOM and not served, mb
        g.close()
    assert served


def _with_lengths(cch, seed):
    """Few distinct times, so that ties occur everywhere, and lengths; INF kept."""
    rng = np.random.default_rng(seed)
    d, ln = dict(cch), []
    for key in ("up_w", "down_w"):
        w = np.asarray(cch[key], np.uint32)
        d[key] = np.where(w == INF, w, rng.integers(0, 4, len(w)).astype(np.uint32))
        ln.append(np.where(w == INF, w, rng.integers(0, 5000, len(w)).astype(np.uint32)))
    return d, ln[0], ln[1]


@pytest.mark.parametrize("name", ["band2", "band16", "band17", "band33", "sources300", "fan"])
def test_panels_two_channel(built, name):
    import bfphast
    up, _, _ = GRAPHS[name]
    n = len(up)
    d, ul, dl = _with_lengths(_cch(n, up, 5, 1, 60, 0.2), 6)
    c = orc.Cch.from_dict(d)
    g = bfphast.Graph.from_cch(d, up_len=ul, down_len=dl)
    rng = np.random.default_rng(n)

    def sets(m):
        return [[(int(rng.integers(0, n)), int(rng.integers(0, 8)), int(rng.integers(0, 500)))
                 for _ in range(int(rng.integers(1, 4)))] for _ in range(m)]

    for S, T in ((1, 1), (33, 40), (70, 9)):
        src, tgt = sets(S), sets(T)
        got = g.matrix_seeded_2ch(src, tgt, with_conflicts=True)
        want = orc.table_phast_lopsided_2ch(c, src, tgt, INF, ul, dl)
        assert all(np.array_equal(a, b) for a, b in zip(got, want)), (S, T)
    for thr in (0, 3, 25, INF):
        seeds = sets(1)[0]
        got, want = g.phast_bounded_seeded_2ch(seeds, thr), c.bounded_seeded_2ch(seeds, thr, ul, dl)
        assert all(np.array_equal(a, b) for a, b in zip(got, want)), thr


def test_panels_two_channel_wide_levels(built, grid100):
    """Levels of more units than blocks (a warp per unit) against the item sweep."""
    import bfphast
    d, ul, dl = _with_lengths(grid100[1], 2)
    n = d["n"]
    rng = np.random.default_rng(8)
    src = [[(int(r), 0, 0)] for r in rng.choice(n, 70, replace=False)]
    tgt = [[(int(r), 1, 1)] for r in rng.choice(n, 3000, replace=False)]
    g = bfphast.Graph.from_cch(d, up_len=ul, down_len=dl)
    got = g.matrix_seeded_2ch(src, tgt)
    g.set_tune(device_schedule=0)
    want = g.matrix_seeded_2ch(src, tgt)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    c = orc.Cch.from_dict(d)
    ref = orc.table_phast_lopsided_2ch(c, src[:4], tgt, INF, ul, dl)
    assert np.array_equal(got[0][:4], ref[0]) and np.array_equal(got[1][:4], ref[1])


@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_plain_sweep_by_panels(built, name):
    """The plain engine's one-launch sweep (panels) and its launch per level
    (rows) against the oracle: partial and whole batches, seeds taken back
    between them, a threshold within the sweep, saturating sums."""
    import bfphast
    up, lo, hi = GRAPHS[name]
    n = len(up)
    cch = _cch(n, up, 7, lo, hi, 0.2)
    c = orc.Cch.from_dict(cch)
    g = bfphast.Graph.from_cch(cch)
    g.set_engine(bfphast.ENGINE_PLAIN)
    rng = np.random.default_rng(n)
    every = np.arange(n, dtype=np.uint32)
    for k in (1, 8, 9, 31, 32, 33, 100):
        src = rng.integers(0, n, k).astype(np.uint32)
        tgt = rng.integers(0, n, 7).astype(np.uint32)
        want, _ = c.matrix(src, every)
        for persist in (1, 0, 1):
            g.set_tune(persistent_sweep=persist)
            assert np.array_equal(g.query_batch(src), want), (k, persist)
            assert np.array_equal(g.matrix(src, tgt), want[:, tgt]), (k, persist)
            for thr in (0, lo, min(INF - 1, 5 * (hi // 2))):
                got = g.matrix(src, tgt, threshold=thr)
                assert np.array_equal(got, np.where(want[:, tgt] <= thr, want[:, tgt], INF)), thr


def test_plain_sweep_of_a_slab_beyond_l2(built):
    """A graph whose plain slab exceeds L2 (the sweep's other launch shape):
    55,000 runs of 20 ranks, each rank joined to the next three of its run."""
    import bfphast
    n, run = 1_100_000, 20
    u = np.arange(n, dtype=np.int64)
    pairs = [np.stack([v := u[(u % run) < run - k], v + k], 1) for k in (1, 2, 3)]
    up = np.concatenate(pairs)
    up = up[np.lexsort((up[:, 1], up[:, 0]))]
    rng = np.random.default_rng(2)
    w = rng.integers(1, 100, (2, len(up))).astype(np.uint32)
    o = np.lexsort((up[:, 0], up[:, 1]))
    off = np.zeros((2, n + 1), np.uint64)
    off[0, 1:] = np.cumsum(np.bincount(up[:, 0], minlength=n))
    off[1, 1:] = np.cumsum(np.bincount(up[:, 1], minlength=n))
    cch = dict(n=n, up_off=off[0], up_tgt=up[:, 1].astype(np.uint32), up_w=w[0],
               down_off=off[1], down_tgt=up[o, 0].astype(np.uint32), down_w=w[1][o])
    g = bfphast.Graph.from_cch(cch)
    g.set_engine(bfphast.ENGINE_PLAIN)
    src = rng.integers(0, n, 33).astype(np.uint32)
    got = g.query_batch(src)
    g.set_tune(persistent_sweep=0)
    assert np.array_equal(got, g.query_batch(src))
    assert ((got != INF).sum(1) == run).all() and (got[np.arange(33), src] == 0).all()
