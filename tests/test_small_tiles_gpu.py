"""Kernels that take other tiles, or other parts of a tile per thread, for few rows: the same sums in the same order, so a row's answer does
not depend on how many others are with it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,d", [(19_500, 300, 130), (19_000, 1_030, 131), (20_001, 257, 355)])
def test_dense_chain_of_few_rows(n, k, d):
    import superkmeans_b200 as skm

    eng = skm.engine
    rng = np.random.default_rng(d)
    c = rng.standard_normal((k, d), dtype=np.float32)
    x = (c[rng.integers(0, k, n)] + np.float32(0.7) * rng.standard_normal((n, d), dtype=np.float32)).astype(np.float32)
    previous = rng.integers(0, k, n).astype(np.uint32)
    first = max(2, eng.dimension_split(d)[1] // 2)
    eng.set_prune_split(2)
    try:
        whole = eng.find_nearest_pruned(x, c, previous, first)
        for lo, hi in ((0, 1), (1, 32), (32, 64), (64, 97), (97, 5_000), (5_000, 5_000 + 128 * 148)):
            piece = eng.find_nearest_pruned(x[lo:hi], c, previous[lo:hi], first)
            for a, b in zip(whole, piece):
                assert (a[lo:hi] == b).all(), (lo, hi)
    finally:
        eng.set_prune_split(0)


@pytest.mark.parametrize("n,d", [(40_000, 33), (9_000, 129), (9_000, 355), (3_000, 770)])
def test_product_of_few_rows(n, d):
    import superkmeans_b200 as skm

    rng = np.random.default_rng(d)
    m, x = rng.standard_normal((d, d), dtype=np.float32), rng.standard_normal((n, d), dtype=np.float32)
    whole = skm.engine.unrotate(m, x)
    want = x.astype(np.float64) @ m.astype(np.float64)
    scale = np.linalg.norm(x, axis=1)[:, None] * np.linalg.norm(m, axis=0)
    assert (np.abs(whole - want) <= d * 2.0 ** -24 * scale).all()   # a rounding per term
    for rows in (1, 31, 32, 33, 65, 900):
        assert (skm.engine.unrotate(m, x[:rows]) == whole[:rows]).all(), rows


@pytest.mark.parametrize("n,k,d", [(2_000, 700, 33), (1_501, 701, 128), (1_300, 1_000, 101), (5_001, 193, 64), (10_000, 65, 100)])
def test_direct_tiles_of_few_rows(n, k, d):
    import superkmeans_b200 as skm

    rng = np.random.default_rng(d)
    x, y = rng.standard_normal((n, d), dtype=np.float32), rng.standard_normal((k, d), dtype=np.float32)
    knn, dist = skm.engine.find_nearest(x, y)
    x64, y64 = x.astype(np.float64), y.astype(np.float64)
    true = (x64 ** 2).sum(1)[:, None] + (y64 ** 2).sum(1) - 2 * x64 @ y64.T
    scale = (x64 ** 2).sum(1) + (y64 ** 2).sum(1).max()
    assert (true[np.arange(n), knn] - true.min(1) <= 2 * d * 2.0 ** -24 * scale).all()   # a rounding per term, for either of two centroids
    assert (np.abs(dist - true[np.arange(n), knn]) <= d * 2.0 ** -24 * scale).all()
    for lo, hi in ((0, 9), (9, 73), (73, 137), (137, 400)):
        a, b = skm.engine.find_nearest(x[lo:hi], y)
        assert (a == knn[lo:hi]).all() and (b == dist[lo:hi]).all(), (lo, hi)
