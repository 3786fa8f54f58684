"""Where a block's search through the grid of bv_knn ends: a third coordinate
that dwarfs the plane, centroids beyond every side and corner of the
locations, locations far from the origin, keys beyond the double range.
Indices and order against findNearestPoints, bit-exact."""
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
    L = [_layout3(bvlib, a, y, z, 100) for a in (x, far)]
    best = [np.inf, np.inf]
    for rep in range(60):  # in turn, the least of each: the machine is shared
        for i in (0, 1):
            t0 = time.perf_counter()
            bvlib.knn(L[i])
            best[i] = min(best[i], time.perf_counter() - t0)
        if rep >= 7 and best[0] <= 1.95 * best[1]:
            break
    assert best[0] <= 1.95 * best[1], best


def _planar(n, cs, g, x, y):
    bn = np.array([cs + 5] + [5] * ((n - cs - 5) // 5), np.int32)
    bn[-1] += n - int(bn.sum())
    acc = np.concatenate([[0], np.cumsum(bn)]).astype(np.int32)
    return bn, acc, x[acc[:-1]].copy(), y[acc[:-1]].copy()


@pytest.mark.parametrize("kind", ["uniform", "clusters"])
@pytest.mark.parametrize("cs", [7, 60])
def test_centroids_outside(bvlib, oracle, kind, cs):
    """Centroids of blocks that search the grid (2,048 earlier locations and
    more) beyond each side and corner: just outside, by a third of the extent
    and far away, and the opposite way round at positions along the sides."""
    g = np.random.default_rng(cs)
    n = 9000
    x, y = g.random(n), g.random(n)
    if kind == "clusters":
        c = g.integers(0, 6, n)
        x = g.random(6)[c] + 0.01 * g.standard_normal(n)
        y = g.random(6)[c] + 0.01 * g.standard_normal(n)
    bn, acc, cx, cy = _planar(n, cs, g, x, y)
    late = np.flatnonzero(acc[:-1] >= 2048)
    moved = g.permutation(late)[:160]
    for t, b in enumerate(moved):
        sx, sy = ((-1, 0), (1, 0), (0, -1), (0, 1), (-1, -1), (-1, 1), (1, -1), (1, 1))[t % 8]
        h = (1e-9, 1e-3, 0.3, 40.0, 1e7)[t // 8 % 5]
        if sx:
            cx[b] = x.max() + h if sx > 0 else x.min() - h
        if sy:
            cy[b] = y.max() + h if sy > 0 else y.min() - h
    assert np.all(acc[moved] >= 2048)
    L = bvlib.Layout(bn, acc, x, y, np.zeros(n), cs, cx, cy)
    assert np.array_equal(bvlib.knn(L), oracle.knn_all_fast(x, y, cs, acc, cx, cy))


@pytest.mark.parametrize("cs", [3, 20, 60])
@pytest.mark.parametrize("e", [41, 44])
def test_far_from_the_origin(bvlib, oracle, cs, e):
    """A unit square at 2^41 (coordinates are multiples of 2^-11, a thirtieth
    of a cell) and 2^44 (a quarter): a window's sides are not representable as
    coordinates."""
    g = np.random.default_rng(cs + e)
    n = 16000
    x, y = g.random(n) + 2.0 ** e, g.random(n) - 2.0 ** e
    bn, acc, cx, cy = _planar(n, cs, g, x, y)
    L = bvlib.Layout(bn, acc, x, y, np.zeros(n), cs, cx, cy)
    assert np.array_equal(bvlib.knn(L), oracle.knn_all_fast(x, y, cs, acc, cx, cy))


def test_keys_beyond_the_double_range(bvlib, oracle):
    """Squared distances that overflow tie at infinity: a third of the
    locations 1e200 away, and some centroids between."""
    g = np.random.default_rng(2)
    n, cs = 6000, 40
    x, y = g.random(n), g.random(n)
    x[g.permutation(n)[:n // 3]] += 1e200
    bn, acc, cx, cy = _planar(n, cs, g, x, y)
    cx[g.permutation(np.flatnonzero(acc[:-1] >= 2048))[:5]] = 5e199
    L = bvlib.Layout(bn, acc, x, y, np.zeros(n), cs, cx, cy)
    assert np.array_equal(bvlib.knn(L), oracle.knn_all_fast(x, y, cs, acc, cx, cy))
