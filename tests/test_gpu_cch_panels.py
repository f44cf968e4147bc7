"""Customization by panels (up to 16 consecutive apexes of a run relaxed
together) against the oracle, bit for bit: runs at and beside the panel, rows
and columns at the edges of their blocks, missing directions and pairs, sums
that saturate, both relaxations, panels above levels of apexes."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu
INF = 0xFFFFFFFF


def _topo(n, pairs, rng, one_way):
    """A topology of the given pairs (u < v), a share of them in one direction
    only, about two thirds of the edges shortcuts."""
    pairs = np.array(sorted(pairs), np.int64).reshape(-1, 2)
    kind = rng.random(len(pairs))
    up = pairs[kind > one_way / 2]
    dn = pairs[(kind < one_way / 2) | (kind > one_way)]
    dn = dn[np.lexsort((dn[:, 0], dn[:, 1]))]
    off = np.zeros((2, n + 1), np.uint64)
    off[0, 1:] = np.cumsum(np.bincount(up[:, 0], minlength=n))
    off[1, 1:] = np.cumsum(np.bincount(dn[:, 1], minlength=n))
    short = [(rng.random(len(x)) < 0.66).astype(np.uint8) for x in (up, dn)]
    mid = [np.where(s, rng.integers(0, n, len(s)), INF).astype(np.uint32) for s in short]
    return orc.CchTopo(n, off[0], up[:, 1].astype(np.uint32), off[1], dn[:, 0].astype(np.uint32),
                       up_short=short[0], down_short=short[1], up_mid=mid[0], down_mid=mid[1])


def _clique(n, base=0):
    return {(base + u, base + v) for u in range(n) for v in range(u + 1, n)}


def _cases():
    # one run: its last panel short or whole, 18 to 84 columns above the first
    for n in (34, 47, 48, 49, 50, 63, 64, 65, 80, 100):
        yield "clique%d" % n, n, _clique(n)
    # columns slide past each other inside a panel
    yield "band", 150, {(u, v) for u in range(150) for v in range(u + 1, min(150, u + 40))}
    # runs below a common top, as the parts of a dissection
    top = _clique(40, 120)
    yield "tree", 160, top | {p for b in (0, 40, 80) for p in _clique(40, b)} | {
        (b + u, 120 + v) for b in (0, 40, 80) for u in range(40) for v in range(0, 40, 2)}
    # rows that are no runs: panels of one row
    yield "stars", 130, {(u, v) for u in range(0, 60) for v in range(60, 130)} | _clique(70, 60)


CASES = {c[0]: c for c in _cases()}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("drop", [0.0, 0.3])  # pairs left out: not closed, runs broken
@pytest.mark.parametrize("w_max", [1000, INF])
def test_relaxations(built, name, drop, w_max):
    import bfphast
    _, n, pairs = CASES[name]
    rng = np.random.default_rng([n, int(drop * 10), w_max & 1])
    pairs = [p for p in sorted(pairs) if rng.random() >= drop]
    t = _topo(n, pairs, rng, 0.3)
    g = bfphast.Cch.from_oracle_topo(t)
    nu, nd = len(t.up_mid), len(t.down_mid)

    def weights(count):
        w = rng.integers(0, w_max, count, dtype=np.uint64).astype(np.uint32)
        w[rng.random(count) < 0.1] = INF
        return w
    for _ in range(2):
        up, dn = weights(nu), weights(nd)
        got, want = g.relax(up, dn, t.up_mid, t.down_mid), t.relax(up, dn)[:4]
        assert all(np.array_equal(a, b) for a, b in zip(got, want))
        lu, ld = weights(nu), weights(nd)
        got = g.relax_lex(up, dn, lu, ld, t.up_mid, t.down_mid)
        want = t.relax_lex(up, dn, lu, ld)[:4]
        assert all(np.array_equal(a, b) for a, b in zip(got, want))
