"""Ids out of range in the device variants: the call that has them fails, and
nothing of it reaches the next one."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _check(cch, S, engine, overlap, ends):
    """Calls whose sources and targets go through `ends`, each followed by a valid one."""
    import torch

    import bfphast
    n = cch["n"]
    g = bfphast.Graph.from_cch(cch)
    g.set_engine(engine)
    g.set_tune(overlap_upward=overlap)
    rng = np.random.default_rng(S)
    src, tgt = (rng.integers(0, n, k).astype(np.uint32) for k in (S, 50))
    want, _ = orc.Cch.from_dict(cch).matrix(src[:40], tgt)
    out = torch.empty(S, 50, dtype=torch.int32, device="cuda")

    def call(s, t):
        d = [torch.from_numpy(x.view(np.int32)).cuda() for x in (s, t)]
        g.matrix_device(d[0].data_ptr(), S, d[1].data_ptr(), 50, out.data_ptr())

    for bad in (n, n + 5, 0xFFFFFFFF):
        with pytest.raises(bfphast.BfError) as e:
            call(*ends(src.copy(), tgt.copy(), bad))
        assert e.value.status == bfphast.BF_ERR_INVALID, bad
        call(src, tgt)
        assert np.array_equal(out[:40].cpu().numpy().view(np.uint32), want), bad


def _last(x, bad):
    x[-1] = bad
    return x


@pytest.mark.parametrize("S", [1, 40, 3000])
@pytest.mark.parametrize("overlap", [1, 0])
@pytest.mark.parametrize("engine", [1, 2])  # plain, batched
def test_invalid_sources(built, grid100, S, overlap, engine):
    _check(grid100[1], S, engine, overlap, lambda s, t, bad: (_last(s, bad), t))


@pytest.mark.parametrize("S", [1, 40, 3000])
@pytest.mark.parametrize("overlap", [1, 0])
@pytest.mark.parametrize("engine", [1, 2])
def test_invalid_targets_beside_invalid_sources(built, grid100, S, overlap, engine):
    """The targets end the call while the sources are still walked."""
    _check(grid100[1], S, engine, overlap, lambda s, t, bad: (_last(s, bad), _last(t, bad)))
    _check(grid100[1], S, engine, overlap, lambda s, t, bad: (s, _last(t, bad)))
