"""Tile emission over row widths and array alignments: four cells a thread
across row ends, wide rows counted from their 16-byte boundary, lists of kept
positions longer than a warp holds, and counts scanned by one block or by
many. Every column compared exactly with the oracle."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

MAX = orc.INF


@pytest.fixture(scope="module")
def bf():
    import bfphast
    bfphast.load()
    return bfphast


def emit(bf, m, src, dst, thr, mask, lat, sparse, shift):
    """Device emission with the matrix, lengths and ids `shift` words off
    their 16-byte boundary."""
    import torch

    def put(a, off=shift):
        buf = torch.zeros(a.size + 4, dtype=torch.int32, device="cuda")
        buf[off:off + a.size] = torch.from_numpy(a.reshape(-1).view(np.int32)).cuda()
        return buf[off:off + a.size]
    n_src, n_dst = m.shape
    dm, ds, dd = put(m), put(src), put(dst)
    dl = None if lat is None else put(lat)
    dmo = dmk = None
    if mask is not None:
        off, flat = orc.mask_csr(mask)
        dmo = torch.from_numpy(off.view(np.int64)).cuda()
        dmk = put(flat, 0)
    cols = [torch.full((m.size,), -7, dtype=torch.int32, device="cuda") for _ in range(4)]
    rows = bf.tile_emit_device(
        dm.data_ptr(), n_src, n_dst, ds.data_ptr(), dd.data_ptr(), [c.data_ptr() for c in cols],
        thr, None if mask is None else dmo.data_ptr(), None if mask is None else dmk.data_ptr(),
        0 if mask is None else len(mask), 0 if mask is None else flat.size,
        None if lat is None else dl.data_ptr(), sparse)
    return tuple(c[:rows].cpu().numpy().view(np.uint32) for c in cols)


@pytest.mark.parametrize("n_dst", [1, 2, 3, 5, 1023, 2047, 2048, 2049, 2050, 2051, 16381, 16382,
                                   16384, 16385, 32769])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
@pytest.mark.parametrize("keep", [0.0, 0.004, 1.0])
def test_widths_and_alignments(bf, n_dst, shift, keep):
    rng = np.random.default_rng([n_dst, shift, int(keep * 1000)])
    n_src = 7
    m = rng.integers(100_001, 200_000, (n_src, n_dst)).astype(np.uint32)
    m[rng.random(m.shape) < keep] = 77_000
    m[rng.random(m.shape) < 0.001] = 5_000_000  # saturates at 1000x
    m[0, -1] = m[-1, 0] = 1  # the ends of rows are kept in any case
    m[rng.random(m.shape) < 0.01] = MAX
    src = rng.permutation(n_src).astype(np.uint32)
    dst = rng.permutation(3 * n_dst)[:n_dst].astype(np.uint32)
    lat = rng.integers(0, 1 << 32, m.shape, dtype=np.uint64).astype(np.uint32)
    mask = [np.flatnonzero(rng.random(3 * n_dst) < p).astype(np.uint32).tolist()
            for p in (0, 1, 0.5, 0.1, 1, 0.9, 0.03)]
    for sparse in (False, True):
        for mk in (None, mask):
            for thr in (100_000, MAX):
                got = emit(bf, m, src, dst, thr, mk, lat, sparse, shift)
                want = orc.tile_emit(m, n_src, n_dst, src, dst, thr, mk, lat, sparse)
                assert all(np.array_equal(a, b) for a, b in zip(got, want)), (sparse, thr)


@pytest.mark.parametrize("n_src", [16384, 16385])  # counts of one block's scan, and one more
@pytest.mark.parametrize("n_dst", [1, 2048])
def test_many_counts(bf, n_src, n_dst):
    rng = np.random.default_rng(n_src + n_dst)
    rows = n_src if n_dst == 2048 else n_src * 2048  # narrow rows: a count per 2048 cells
    m = rng.integers(0, 1000, (rows, n_dst), dtype=np.uint32)
    src, dst = np.arange(rows, dtype=np.uint32), np.arange(n_dst, dtype=np.uint32)
    got = emit(bf, m, src, dst, 3, None, None, True, 0)
    si, di = np.nonzero(m <= 3)
    want = (si, di, m[si, di] * 1000, np.full(len(si), MAX))
    assert all(np.array_equal(a, b.astype(np.uint32)) for a, b in zip(got, want))
