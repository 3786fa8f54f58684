"""The streamed kernel's CTA shapes at the block sizes where a tile, a panel or
the shape changes, in launches large enough for each shape's rule (more than
two blocks per SM), both sides of the rules' block counts, and the largest
blocks of the kernel.

Tolerance: 1e-10 relative on the total log-likelihood, the FP64 parity bound;
per block 1e-8 of max(1, |value|): with a nugget of 0.05 the condition numbers
stay below (M + 0.05) / 0.05 < 2e4, so that M rounded updates per entry move a
block by less than 2e4 x 820 x 2^-53 = 2e-9 of its size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REL = 1e-10
W96, W160, W256, W128, W160_2, ONE_WARP = 0, 1, 2, 3, 4, 5  # streamed_variant
ODD = [1, 2, 7, 8, 9, 15, 16, 17]


def _layout(bv, sizes, cs, seed=0):
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


def _check(bv, oracle, L, theta, variant, nugget=0.05):
    P = oracle.OracleProblem(L.batchNum, L.batchNumAccum, L.x, L.y, L.obs, L.knn_idx, L.cs, 1.0,
                             nugget=nugget)
    ref, pb = oracle.llh(P, theta, per_block=True)
    per = -(pb[:, 1] ** 2 + pb[:, 0] + L.batchNum * np.log(2 * 3.141592653589793)) * 0.5
    with bv.LlhData(L, nugget=True, schedule="streamed") as D:
        v = D(tuple(theta) + (nugget,))
        bl = D.block_llk()
        st = D.status()
    assert st["failed"] == 0 and st["streamed_blocks"] == L.bc
    assert st["streamed_variant"] == variant
    assert abs(v - ref) <= REL * abs(ref), (v, ref)
    assert np.all(np.abs(bl - per) <= 1e-8 * np.maximum(1.0, np.abs(per)))
    return bl


@pytest.mark.parametrize("nu", [0.5, 1.5, 0.8])
@pytest.mark.parametrize("cs,variant", [(49, W96), (63, W96), (68, W96), (69, W128), (95, W128), (112, W128),
                                        (168, W128), (169, W160), (191, W160), (224, W160), (233, W160),
                                        (234, W256), (271, W256)])
def test_shapes_of_large_launches(bvlib, oracle, cs, variant, nu):
    """Block sizes around the tiles' and panels' edges on each shape; the
    launches of at most two blocks per SM, half the blocks each, give the same
    bits on theirs."""
    L = _layout(bvlib, [cs] + ODD * 40, cs, seed=cs)
    th = (1.1, 0.15, nu)
    bl = _check(bvlib, oracle, L, th, variant)
    for shard in (0, 1):
        with bvlib.LlhData(L, nugget=True, shard_count=2, shard_index=shard) as S:
            S(th + (0.05,))
            assert S.status()["streamed_variant"] == (W256 if cs + 17 > 250 else W160_2)
            mine = bvlib.shard_blocks(L.batchNum, cs, 2, shard)
            assert np.array_equal(S.block_llk()[mine], bl[mine])


@pytest.mark.parametrize("nu,blocks,variant", [(0.5, 296, W160_2), (0.5, 297, W96), (0.8, 296, W160_2),
                                               (0.8, 297, W96), (0.5, 591, W96), (0.5, 592, ONE_WARP),
                                               (0.8, 592, W96)])
def test_block_counts(bvlib, oracle, nu, blocks, variant):
    """The counts at which small blocks (M <= 48) change shape."""
    L = _layout(bvlib, [40] + [1 + i % 9 for i in range(blocks - 1)], 30, seed=blocks)
    _check(bvlib, oracle, L, (1.0, 0.2, nu), variant)


@pytest.mark.parametrize("nu", [0.5, 0.8])
@pytest.mark.parametrize("cs", [769, 770, 783, 802])
def test_largest_blocks(bvlib, oracle, cs, nu):
    """Blocks up to the kernel's largest (M = 819); for a general nu up to and
    beyond the last whose table window has room in shared memory (M = 786)."""
    L = _layout(bvlib, [cs] + [17, 16, 1, 9], cs, seed=cs)
    _check(bvlib, oracle, L, (1.0, 0.2, nu), W256)


def test_beyond_the_largest_block(bvlib):
    L = _layout(bvlib, [803, 17], 803)
    with pytest.raises(bvlib.BvError):
        bvlib.LlhData(L, schedule="streamed")
