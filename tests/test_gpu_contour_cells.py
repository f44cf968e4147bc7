"""Cells of contour rasters, whose indices are found without a division where
that is certain: points on and next to cell borders, far from and below the
origin, cell sizes without an exact reciprocal, and sizes out of its range;
against floor((x - origin) / cell) in double precision."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cells(xy, cell):
    o = xy.min(0) - cell * 3.0
    c = np.floor((xy - o) / cell).astype(np.int64)
    return {tuple(v) for v in c}, tuple(o)


@pytest.mark.parametrize("cell", [30.0, 200.1, 1.0, 1.0 / 3, 0.1, 1e-3, 6.67e2, 1e5])
@pytest.mark.parametrize("span", [0, 40, 3000])
def test_borders(built, cell, span):
    import bfphast
    rng = np.random.default_rng([int(cell * 1000), span])
    lo = np.array([4.8e5, -6.58e6])
    k = rng.integers(0, span + 1, (4000, 2)).astype(float)
    xy = lo + k * cell  # on the borders the origin's own rounding gives, or a step off them
    for step in range(-2, 3):
        pick = slice(step + 2, None, 6)
        for _ in range(abs(step)):
            xy[pick] = np.nextafter(xy[pick], np.sign(step) * np.inf)
    xy[5::6] += rng.random(xy[5::6].shape) * cell
    xy[0] = lo
    want, o = _cells(xy, cell)
    got = bfphast.contour_rasters([{"segments": [p[None] for p in xy], "cell_m": cell}], 0, 0)
    cells, origin = got[0]
    assert tuple(origin) == o
    assert {tuple(v) for v in np.asarray(cells).tolist()} == want


@pytest.mark.parametrize("cell", [1e290, 5e307])
def test_cell_sizes_without_a_normal_reciprocal(built, cell):
    import bfphast
    xy = np.array([[0.0, 0.0], [5.0, 7.0], [1.0, -3.0]])
    want, _ = _cells(xy, cell)
    got = bfphast.contour_rasters([{"segments": [xy[:1], xy[1:2], xy[2:]], "cell_m": cell}], 0, 0)
    assert {tuple(v) for v in np.asarray(got[0][0]).tolist()} == want


def test_lines_between_far_cells(built):
    """Segments across words, steep, flat, backward and closed on themselves: the
    cells of a line drawn over each pair of points."""
    import bfphast
    rng = np.random.default_rng(3)
    segs = [rng.integers(0, 200, (n, 2)) * 30.0 + 15.0 for n in (2, 3, 5, 2, 9, 40)]
    segs += [np.array([[15.0, 15.0], [15.0, 15.0]]), np.array([[15.0, 6000.0], [6000.0, 15.0]])]
    lo = np.concatenate(segs).min(0) - 90.0
    want = set()
    for s in segs:
        c = np.floor((s - lo) / 30.0).astype(int)
        want.add(tuple(c[0]))
        for (c0, r0), (c1, r1) in zip(c[:-1].tolist(), c[1:].tolist()):
            dx, dy = abs(c1 - c0), abs(r1 - r0)
            sx, sy, e = (1 if c0 < c1 else -1), (1 if r0 < r1 else -1), dx - dy
            while True:
                want.add((c0, r0))
                if (c0, r0) == (c1, r1):
                    break
                e2 = 2 * e
                if e2 > -dy:
                    e, c0 = e - dy, c0 + sx
                if e2 < dx:
                    e, r0 = e + dx, r0 + sy
    got = bfphast.contour_rasters([{"segments": segs, "cell_m": 30.0}], 0, 0)
    assert {tuple(v) for v in np.asarray(got[0][0]).tolist()} == want
