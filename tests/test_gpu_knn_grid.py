"""Conditioning sets through the grid (bv_knn for layouts of 4,096 locations
and more) against findNearestPoints: indices and order bit-exact on location
sets that stretch, cluster or degenerate the grid, with ties, with centroids
outside the locations' box, and for a third coordinate."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(kind, n, g):
    if kind == "uniform":
        return g.random(n), g.random(n)
    if kind == "strip":      # one row of cells
        return g.random(n), 1e-4 * g.random(n)
    if kind == "line":       # no extent in y
        return g.random(n), np.full(n, 0.25)
    if kind == "one":        # no extent at all: everything tied
        return np.full(n, -3.0), np.full(n, 7.0)
    if kind == "lattice":    # exact ties everywhere
        i = g.permutation(n)
        m = int(np.ceil(np.sqrt(n)))
        return (i % m) / 64.0, (i // m) / 64.0
    c = g.random((8, 2)) * 1e3 - 500  # clusters, far apart, and one outlier
    s = 10.0 ** g.uniform(-4, 1, 8)
    k = g.integers(0, 8, n)
    p = c[k] + g.standard_normal((n, 2)) * s[k, None]
    p[0] = (1e6, -1e6)
    return p[:, 0].copy(), p[:, 1].copy()


def _blocks(n, cs, g, sorted_by=None):
    sizes = [cs + 5]
    while sum(sizes) < n:
        sizes.append(int(min(g.integers(1, 40), n - sum(sizes))))
    bn = np.asarray(sizes, dtype=np.int32)
    return bn, np.concatenate([[0], np.cumsum(bn)]).astype(np.int32)


def _centroids(p, acc):
    return np.add.reduceat(p, acc[:-1]) / np.diff(acc)


@pytest.mark.parametrize("kind,n,cs", [("uniform", 12000, 100), ("uniform", 4096, 1), ("uniform", 9000, 512),
                                       ("strip", 9000, 60), ("line", 9000, 60), ("lattice", 10000, 77),
                                       ("clusters", 12000, 129)])
@pytest.mark.parametrize("order", ["random", "sorted"])
def test_grid_against_oracle(bvlib, oracle, kind, n, cs, order):
    g = np.random.default_rng(n + cs)
    x, y = _points(kind, n, g)
    if order == "sorted":  # the prefix fills the domain from one side
        i = np.lexsort((y, x))
        x, y = x[i].copy(), y[i].copy()
    bn, acc = _blocks(n, cs, g)
    cx, cy = _centroids(x, acc), _centroids(y, acc)
    cx[3], cy[3] = x.max() + 10.0, y.min() - 1.0  # outside the box, in its corner
    cx[-1], cy[-1] = x.max() + 1e-3, y.max()
    L = bvlib.Layout(bn, acc, x, y, np.zeros(n), cs, cx, cy)
    got = bvlib.knn(L)
    ref = oracle.knn_all_fast(x, y, cs, acc, cx, cy)
    assert np.array_equal(got, ref)


def test_grid_all_points_equal(bvlib, oracle):
    """Every location equal: the grid is one cell and every key a tie."""
    g = np.random.default_rng(0)
    n, cs = 5000, 20
    x, y = _points("one", n, g)
    bn = np.array([4990, 4, 6], np.int32)
    acc = np.array([0, 4990, 4994, 5000], np.int32)
    cx, cy = _centroids(x, acc), _centroids(y, acc)
    L = bvlib.Layout(bn, acc, x, y, np.zeros(n), cs, cx, cy)
    assert np.array_equal(bvlib.knn(L), oracle.knn_all(x, y, cs, acc, cx, cy))


@pytest.mark.parametrize("slots", [3, 40])
def test_grid_third_coordinate(bvlib, oracle, slots):
    """Locations repeated over time slots (ties in the 3-D key)."""
    x, y, z = bvlib.generate_xyt(6000 // slots, slots, 1)
    n, cs = len(x), 90
    g = np.random.default_rng(slots)
    i = g.permutation(n)
    x, y, z = x[i].copy(), y[i].copy(), z[i].copy()
    bn, acc = _blocks(n, cs, g)
    c = [_centroids(p, acc) for p in (x, y, z)]
    L = bvlib.Layout(bn, acc, x, y, np.zeros(n), cs, c[0], c[1], z=z, cz=c[2])
    got = bvlib.knn(L)
    for b in list(range(1, 12)) + list(range(len(bn) - 60, len(bn))):
        ref = oracle.knn_block3_fast(x, y, z, int(acc[b]), c[0][b], c[1][b], c[2][b], cs)
        assert np.array_equal(got[b * cs:(b + 1) * cs], ref), b
