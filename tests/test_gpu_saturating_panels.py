"""Panel sweeps in the saturating form of the relaxation (labels or seed costs
past 2^31) in wide levels: every shape of lane block, and the ring of bulk
copies, against the item sweep (the same u32 results, tolerance 0) and, on a few
sources, the oracle."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu
INF = 0xFFFFFFFF


def _scaled(cch, by):
    """The graph with every finite weight multiplied, at most INF - 1."""
    d = dict(cch)
    for k in ("up_w", "down_w"):
        w = np.asarray(cch[k], np.uint32)
        d[k] = np.where(w == INF, w, np.minimum(w.astype(np.uint64) * by, INF - 1)).astype(np.uint32)
    return d


# labels below 2^31 under a bound past it (the longest path), past it, saturating
@pytest.mark.parametrize("by", [4000, 150000, 300000])
@pytest.mark.parametrize("S", [3, 33, 65, 70, 128, 130, 520, 1030])
def test_labels_past_the_short_range(built, grid100, by, S):
    import bfphast
    cch = _scaled(grid100[1], by)
    n = cch["n"]
    rng = np.random.default_rng(S)
    src = rng.integers(0, n, S).astype(np.uint32)
    tgt = np.arange(0, n, 2, dtype=np.uint32)
    g = bfphast.Graph.from_cch(cch)
    got = g.matrix(src, tgt)
    cut = g.matrix(src, tgt, threshold=0x90000000)
    g.set_tune(device_schedule=0)
    assert np.array_equal(got, g.matrix(src, tgt))
    assert np.array_equal(cut, np.where(got <= 0x90000000, got, INF))
    assert by == 4000 or (got[got != INF] > 0x7FFFFFFF).any()
    want, _ = orc.Cch.from_dict(cch).matrix(src[:3], tgt)
    assert np.array_equal(got[:3], want)


@pytest.mark.parametrize("S", [33, 70, 130, 520])
def test_seed_costs_past_the_short_range(built, grid100, S):
    """On a graph whose own labels fit: absent edges weigh 2^31 - 1 in its tiles."""
    import bfphast
    cch = grid100[1]
    n = cch["n"]
    rng = np.random.default_rng(S)
    costs = np.concatenate([rng.integers(0, 500, S), rng.integers(1 << 31, INF, S),
                            rng.integers(INF - 3000, INF, S)])
    src = [[(int(rng.integers(0, n)), int(rng.choice(costs)))
            for _ in range(int(rng.integers(1, 3)))] for _ in range(S)]
    tgt = [[(int(r), 0)] for r in range(0, n, 5)]
    g = bfphast.Graph.from_cch(cch)
    got = g.matrix_seeded(src, tgt)
    g.set_tune(device_schedule=0)
    assert np.array_equal(got, g.matrix_seeded(src, tgt))
    few = src[:3]
    c = orc.Cch.from_dict(cch)
    assert np.array_equal(got[:3], orc.table_phast_lopsided(c, few, tgt, INF)[0])
