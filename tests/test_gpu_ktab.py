"""Entries of the general-nu covariance as the streamed kernel evaluates them,
one by one: blocks of one point that condition on one point (cs = 1).  With
nugget 3 and sigma2 = 1 the diagonal is 4, so that a block's value
    -(u^2 + log v + log 2 pi) / 2,   v = 4 - rho^2 / 4,  u = -rho z / (4 sqrt(v))
is that of its one covariance rho to a few roundings; the neighbour's
observation z = 1e25 makes u^2 the whole of it for any rho above 1e-18."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pairs(bv, d):
    """A point at the origin and one block for each distance of d."""
    n = len(d) + 1
    obs = np.zeros(n)
    obs[0] = 1e25
    return bv.Layout(np.ones(n, np.int32), np.arange(n + 1, dtype=np.int32), np.concatenate([[0.0], d]),
                     np.zeros(n), obs, 1, knn_idx=np.zeros(n, np.int32))


def _values(bv, d, theta, schedule, **kw):
    with bv.LlhData(_pairs(bv, d), nugget=True, schedule=schedule, on_failure="continue", **kw) as D:
        D(tuple(theta) + (3.0,))
        return D.block_llk()[1:]


@pytest.mark.parametrize("nu", [50.0, 55.0, 57.0, 60.0, 80.0, 150.0])
def test_large_orders(bvlib, nu):
    """Orders at which con r^nu or K_nu(r) leaves the double range within the
    table's reach: the streamed kernel's entries are those of the persistent
    kernel, which evaluates each directly, not-finite ones included.
    Tolerance: the exponent nu log r of magnitude up to 700 is rounded at
    each side (700 x 2^-52 = 1.6e-13, doubled by the square)."""
    d = np.sort(np.exp(np.random.default_rng(1).uniform(np.log(1e-4), np.log(2.0), 4000)))
    a = _values(bvlib, d, (1.0, 1.0, nu), "streamed")
    b = _values(bvlib, d, (1.0, 1.0, nu), "persistent")
    assert np.array_equal(np.isfinite(a), np.isfinite(b))
    f = np.isfinite(b)
    assert np.all(np.abs(a[f] - b[f]) <= 1e-12 * np.abs(b[f]))


@pytest.mark.parametrize("nu", [0.05, 0.4, 0.8, 1.0, 1.2, 2.2, 6.0, 25.0])
def test_entries(bvlib, nu):
    """Entries at distances below, in and beyond the table's regions and at
    their intervals' ends, against 40 digits.  Tolerance: the direct
    evaluation's roundings (exp(-r): r; exp(nu log r): nu |log r|; two per step
    of the recurrence; some sixteen in the series and the factors), three times
    for the intervals over which the value falls by up to e, twice for the
    square, plus the block's own few."""
    mp = pytest.importorskip("mpmath")
    g = np.random.default_rng(int(100 * nu))
    d = np.exp(g.uniform(np.log(5e-5), np.log(33.0), 220))
    s = 128.0 * 2.0 ** g.integers(-33, 4, 80) * (1 + g.integers(0, 16, 80) / 16)  # interval ends in d^2
    d = np.concatenate([d, np.sqrt(s) * (1 + 2.0 ** -20 * g.integers(-1, 2, 80))])
    d = np.float32(d).astype(np.float64)  # d * d is exact
    got = _values(bvlib, d, (1.0, 1.0, nu), "streamed")
    with mp.workdps(40):
        n, two_pi = mp.mpf(nu), 2 * mp.mpf(3.141592653589793)
        con = 1 / (mp.power(2, n - 1) * mp.gamma(n))
        for k, r in enumerate(map(float, d)):
            rho = con * mp.mpf(r) ** n * mp.besselk(n, mp.mpf(r))
            v = 4 - rho * rho / 4
            u = rho * mp.mpf(1e25) / 4
            ref = -(u * u / v + mp.log(v) + mp.log(two_pi)) / 2
            tol = 2 * (3 * (16 + r + nu * abs(np.log(r)) + 4 * nu) + 8) * 2.0 ** -53
            assert abs((mp.mpf(float(got[k])) - ref) / ref) <= tol, (nu, r)
