"""bv_opts.tune over both kinds of evaluation: the closed forms' kernels and
those of a general nu are tuned each on its own first evaluation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _layout(bv, sizes, cs, seed):
    g = np.random.default_rng(seed)
    bn = np.asarray(sizes, dtype=np.int32)
    acc = np.concatenate([[0], np.cumsum(bn)]).astype(np.int32)
    n = int(acc[-1])
    knn = np.zeros((len(bn), cs), dtype=np.int32)
    knn[0] = np.arange(cs)
    for b in range(1, len(bn)):
        knn[b] = g.integers(0, acc[b] - cs, 1) + np.arange(cs)
    return bv.Layout(bn, acc, g.random(n), g.random(n), g.standard_normal(n), cs, knn_idx=knn.ravel())


@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("order", [(0.5, 0.8), (0.8, 0.5)])
@pytest.mark.parametrize("cs,bs", [(30, 1), (60, 8)])
def test_each_kind_of_nu_is_tuned(bvlib, cs, bs, order, use_graph):
    """Small blocks, where the fastest variants of the two kinds differ (one
    warp per block for the closed forms only): each kind's times are its own,
    its variant is the fastest of them, the other kind's is not touched, and
    the values are the untuned handle's."""
    L = _layout(bvlib, [cs + 4] + [bs] * 20000, cs, cs)
    seen = {}
    with bvlib.LlhData(L, nugget=True, use_graph=use_graph) as P, \
            bvlib.LlhData(L, nugget=True, use_graph=use_graph, tune=True) as D:
        for nu in order + order:
            th = (1.0, 0.1, nu, 0.1)
            assert D(th) == P(th)
            assert np.array_equal(D.block_llk(), P.block_llk())
            st = D.status()
            ms = st["tune_ms"]
            assert all(m > 0 for m in ms)
            assert st["streamed_variant"] == int(np.argmin(ms))
            assert seen.setdefault(nu, ms) == ms
        assert seen[0.5] != seen[0.8]


def test_tuned_with_a_third_coordinate(bvlib):
    """With a third coordinate one kernel serves every nu and is tuned once."""
    x, y, z = bvlib.generate_xyt(300, 10, 0)
    g = np.random.default_rng(0)
    L = _layout(bvlib, [70] + [7] * 418, 60, 3)
    L.x, L.y, L.z = x[:L.n].copy(), y[:L.n].copy(), z[:L.n] + 1e-3 * g.random(L.n)
    with bvlib.LlhData(L, nugget=True) as P, bvlib.LlhData(L, nugget=True, tune=True) as D:
        first = None
        for nu in (0.5, 0.8, 1.5):
            th = (1.0, 0.1, nu, 0.1)
            assert D(th) == P(th)
            first = first or D.status()["tune_ms"]
            assert D.status()["tune_ms"] == first
