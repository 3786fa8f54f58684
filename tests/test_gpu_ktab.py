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
