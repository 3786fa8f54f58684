"""Where a block's search through the grid of bv_knn ends: a third coordinate
that dwarfs the plane.  Indices and order against findNearestPoints, bit-exact."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _groups(n, g, depth):
    """Groups of ten neighbouring points, a third coordinate of `depth`."""
    rep = lambda v: np.repeat(v, 10)  # noqa: E731
    return (rep(g.random(n // 10)) + 1e-4 * g.random(n), rep(g.random(n // 10)) + 1e-4 * g.random(n),
            rep(g.random(n // 10)) * depth)


def _layout3(bv, x, y, z, cs):
    n = len(x)
    bn = np.array([200] + [10] * ((n - 200) // 10), np.int32)
    acc = np.concatenate([[0], np.cumsum(bn)]).astype(np.int32)
    c = [np.add.reduceat(v, acc[:-1]) / bn for v in (x, y, z)]
    return bv.Layout(bn, acc, x, y, np.zeros(n), cs, c[0], c[1], z=z, cz=c[2])


@pytest.mark.parametrize("depth", [1.0, 30.0, 1000.0])
def test_deep_third_coordinate(bvlib, oracle, depth):
    """Windows of the plane that say little or nothing about the 3-D key."""
    g = np.random.default_rng(int(depth))
    x, y, z = _groups(20000, g, depth)
    L = _layout3(bvlib, x, y, z, 90)
    got = bvlib.knn(L)
    for b in list(range(150, 1980, 61)) + list(range(1940, 1981)):
        ref = oracle.knn_block3_fast(x, y, z, int(L.batchNumAccum[b]), L.cx[b], L.cy[b], L.cz[b], 90)
        assert np.array_equal(got[b * 90:(b + 1) * 90], ref), b


def test_deep_third_coordinate_cost(bvlib):
    """Where no window can end the search, windows and prefix together hold at
    most one and a half prefixes: against a call whose locations all fall into
    one cell (an outlier at 1e12), which scans every prefix once.  With windows
    of up to the prefix each the ratio was 2.4; the bound lies between."""
    g = np.random.default_rng(0)
    x, y, z = _groups(300000, g, 1000.0)
    far = x.copy()
    far[0] = 1e12
    best = []
    for a in (x, far):
        L = _layout3(bvlib, a, y, z, 100)
        bvlib.knn(L)
        t = []
        for _ in range(9):
            t0 = time.perf_counter()
            bvlib.knn(L)
            t.append(time.perf_counter() - t0)
        best.append(min(t))
    assert best[0] <= 1.95 * best[1], best
