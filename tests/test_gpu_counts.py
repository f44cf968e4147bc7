"""Row and edge counts of a schedule (bf_stats, bf_schedule_levels) when the
count's own bounded wait runs out: the call that asked for them fails, later
calls are served, and what they report is right.

The wait is made to run out as in the other deadline tests: with
BF_TEST_WITHHOLD_ARRIVAL set, the counting launch runs on two blocks of which
block 1 leaves before its first barrier arrival."""
import contextlib
import os

import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu
INF = 0xFFFFFFFF


@contextlib.contextmanager
def _withheld():
    os.environ["BF_TEST_WITHHOLD_ARRIVAL"] = "1"
    try:
        yield
    finally:
        del os.environ["BF_TEST_WITHHOLD_ARRIVAL"]


def _timeout(call):
    import bfphast
    with _withheld(), pytest.raises(bfphast.BfError) as e:
        call()
    assert e.value.status == bfphast.BF_ERR_TIMEOUT


def _graphs(cch, **kw):
    import bfphast
    g, host = bfphast.Graph.from_cch(cch, **kw), bfphast.Graph.from_cch(cch, **kw)
    host.set_tune(device_schedule=0)
    return g, host


def test_counts_after_a_timeout(built, country_small):
    _, cch = country_small
    g, host = _graphs(cch)
    rng = np.random.default_rng(3)
    src = rng.integers(0, cch["n"], 20).astype(np.uint32)
    tgt = rng.choice(cch["n"], 3000, replace=False).astype(np.uint32)
    _timeout(lambda: g.matrix(src, tgt))
    want, sh = host.matrix(src, tgt, stats=True)
    for _ in range(3):  # the same targets: the schedule is kept, the count is not
        got, sg = g.matrix(src, tgt, stats=True)
        assert np.array_equal(got, want)
        assert (sg["swept_nodes"], sg["swept_edges"]) == (sh["swept_nodes"], sh["swept_edges"])


def test_seeded_calls_report_a_timeout(built, country_small):
    """One and two channels; the call after a failed one is not affected."""
    _, cch = country_small
    ln = [np.where(cch[k] == INF, cch[k], cch[k] // 2 + 1) for k in ("up_w", "down_w")]
    g, host = _graphs(cch, up_len=ln[0], down_len=ln[1])
    n = cch["n"]
    rng = np.random.default_rng(4)
    c = orc.Cch.from_dict(cch)
    one = [[(int(r), 3)] for r in rng.choice(n, 3000, replace=False)]
    two = [[(int(r), 3, 5)] for r in rng.choice(n, 3000, replace=False)]
    src = rng.integers(0, n, 5).astype(np.uint32)
    tgt = rng.integers(0, n, 50).astype(np.uint32)
    want, _ = c.matrix(src, tgt)
    for call in (lambda x: x.matrix_seeded(one[:6], one), lambda x: x.matrix_seeded_2ch(two[:6], two)):
        _timeout(lambda: call(g))
        assert np.array_equal(g.matrix(src, tgt), want)
        assert np.array_equal(call(g), call(host))


def test_level_table_after_a_timeout(built, country_small):
    """bf_schedule_levels of a schedule over panels selects the rows on its own."""
    _, cch = country_small
    g, host = _graphs(cch)
    rng = np.random.default_rng(5)
    src = rng.integers(0, cch["n"], 4).astype(np.uint32)
    tgt = rng.choice(cch["n"], 400, replace=False).astype(np.uint32)
    want = host.matrix(src, tgt)
    assert np.array_equal(g.matrix(src, tgt), want)
    _timeout(g.schedule_levels)
    for a, b in zip(g.schedule_levels(), host.schedule_levels()):
        assert np.array_equal(a, b)
    assert np.array_equal(g.matrix(src, tgt), want)
