"""The streamed kernel's panels at the sizes where a tile, a panel or a CTA
size changes: every block size around the multiples of 8 and 16 rows, the
largest of each CTA size's range, and launches of few and of many blocks.

Tolerance: 1e-10 relative on the total log-likelihood, the FP64 parity bound;
per block 1e-8 of max(1, |value|): nu = 0.5 on these layouts keeps the
condition numbers below ~1e5, a thousand times the rounding of one entry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REL = 1e-10


def _layout(bv, sizes, cs, seed=0):
    """Blocks of the given sizes (block 0 first), random locations and sets."""
    g = np.random.default_rng(seed)
    bn = np.asarray(sizes, dtype=np.int32)
    acc = np.concatenate([[0], np.cumsum(bn)]).astype(np.int32)
    n = int(acc[-1])
    knn = np.zeros((len(bn), cs), dtype=np.int32)
    if cs:
        knn[0] = np.arange(cs)
        for b in range(1, len(bn)):
            knn[b] = g.choice(acc[b], cs, replace=False)
    return bv.Layout(bn, acc, g.random(n), g.random(n), g.standard_normal(n), cs, knn_idx=knn.ravel())


def _check(bv, oracle, L, theta, dist_scale=1.0, nugget=0.0):
    P = oracle.OracleProblem(L.batchNum, L.batchNumAccum, L.x, L.y, L.obs, L.knn_idx, L.cs, dist_scale,
                             nugget=nugget)
    ref, pb = oracle.llh(P, theta, per_block=True)
    per = -(pb[:, 1] ** 2 + pb[:, 0] + L.batchNum * np.log(2 * 3.141592653589793)) * 0.5
    with bv.LlhData(L, dist_scale=dist_scale, nugget=nugget > 0, schedule="streamed") as D:
        v = D(tuple(theta) + ((nugget,) if nugget > 0 else ()))
        bl = D.block_llk()
        assert D.status()["failed"] == 0
    assert abs(v - ref) <= REL * abs(ref), (v, ref)
    assert np.all(np.abs(bl - per) <= 1e-8 * np.maximum(1.0, np.abs(per)))


@pytest.mark.parametrize("nu", [0.5, 1.5, 0.8])
def test_every_block_size(bvlib, oracle, nu):
    """cs = 0, one block of every size from 1 to 67: every remainder of rows
    and columns in a tile and a panel."""
    _check(bvlib, oracle, _layout(bvlib, list(range(1, 68)), 0), (1.2, 0.3, nu))


@pytest.mark.parametrize("cs", [1, 15, 16, 17, 31, 95, 115, 160, 233, 249, 310])
def test_panel_edges(bvlib, oracle, cs):
    """Conditioned blocks whose panels end at, before and after multiples of
    16, across the CTA sizes' ranges, with a nugget and a distance scale."""
    L = _layout(bvlib, [cs + 3] + [1, 2, 7, 8, 9, 15, 16, 17] * 2, cs, seed=cs)
    _check(bvlib, oracle, L, (1.0, 0.2, 0.5))
    _check(bvlib, oracle, L, (0.7, 0.1, 1.5), dist_scale=2.0, nugget=0.05)


@pytest.mark.parametrize("blocks", [440, 450, 590, 600])
def test_few_and_many_small_blocks(bvlib, oracle, blocks):
    """Both sides of the block count at which small blocks change CTA size."""
    L = _layout(bvlib, [40] + [1 + i % 9 for i in range(blocks - 1)], 30, seed=blocks)
    _check(bvlib, oracle, L, (1.0, 0.2, 0.5))


@pytest.mark.parametrize("cs", [0, 1, 14, 15, 16, 31])
@pytest.mark.parametrize("nu", [0.5, 1.5, 2.5])
def test_one_warp_per_block(bvlib, oracle, cs, nu):
    """Launches of small blocks (M <= 48), one block per warp: every size up to
    three full panels, empty blocks between, and the bits of a launch of few
    blocks (CTAs per block)."""
    top = 48 - cs
    L = _layout(bvlib, [max(cs, 20)] + [1 + i % top for i in range(640)] + [0, 3, 0], cs, seed=cs)
    _check(bvlib, oracle, L, (1.1, 0.15, nu), nugget=0.02)
    th = (1.1, 0.15, nu, 0.02)
    with bvlib.LlhData(L, nugget=True) as D, bvlib.LlhData(L, nugget=True, shard_count=3) as S:
        D(th), S(th)
        mine = bvlib.shard_blocks(L.batchNum, cs, 3, 0)
        assert np.array_equal(D.block_llk()[mine], S.block_llk()[mine])


@pytest.mark.parametrize("nu", [0.3, 0.8, 2.2])
@pytest.mark.parametrize("range_", [1e-5, 0.003, 0.1, 30.0])
def test_general_nu_table(bvlib, oracle, nu, range_):
    """A general nu through the table: scaled distances within its regions,
    below, between and beyond them (locations 1e-6 to 1.4 apart, ranges over
    six decades), repeated locations, blocks smaller than a panel."""
    g = np.random.default_rng(7)
    L = _layout(bvlib, [33] + [1, 2, 5, 17, 30] * 4, 30, seed=3)
    # Groups of points 1e-6, 1e-4 and 1e-2 apart around the first ones; the
    # nugget keeps their covariances regular.
    for k, h in enumerate((1e-6, 1e-4, 1e-2, 0.0)):
        i = g.choice(L.n // 2, 12, replace=False)
        L.x[L.n // 2 + 12 * k:L.n // 2 + 12 * (k + 1)] = L.x[i] + h * g.random(12)
        L.y[L.n // 2 + 12 * k:L.n // 2 + 12 * (k + 1)] = L.y[i]
    _check(bvlib, oracle, L, (1.1, range_, nu), nugget=0.1)
    _check(bvlib, oracle, L, (1.1, range_ / 2, nu), dist_scale=2.0, nugget=0.1)
