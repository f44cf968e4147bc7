"""The autotuner on tables that are swept over panels: block size and work items,
which such a sweep does not have, keep the graph's own settings, and a schedule
over panels outlives a change of them."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def test_settings_of_items_stay(built, grid100):
    import torch

    import bfphast
    import workload
    _, cch = grid100
    g = bfphast.Graph.from_cch(cch)
    keep = dict(threads_per_block=256, edges_per_item=24, small_level_rows=96,
                small_level_edges=5)
    g.set_tune(**keep)
    src, tgt = workload.sources_targets(cch["n"], 300, 500, seed=77)
    d_s = torch.from_numpy(src.view(np.int32)).cuda()
    d_t = torch.from_numpy(tgt.view(np.int32)).cuda()
    best = g.autotune(d_s.data_ptr(), len(src), d_t.data_ptr(), len(tgt), reps=1)
    assert best["step_ms"] > 0 and best["lanes_per_wave"] in (0, 160)
    for k, v in keep.items():
        assert best[k] == v and g.get_tune()[k] == v, k
    want, _ = orc.Cch.from_dict(cch).matrix(src[:20], tgt)
    for edges in (24, 8):
        g.set_tune(edges_per_item=edges)
        assert np.array_equal(g.matrix(src, tgt)[:20], want)
    # by items the settings are what is tuned
    g.set_tune(device_schedule=0)
    for edges in (24, 8):
        g.set_tune(edges_per_item=edges)
        assert np.array_equal(g.matrix(src, tgt)[:20], want)
