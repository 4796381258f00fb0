"""First ADSampling test on the tensor cores, the walk over its lists and the dense chain, at the edges of their tiles."""
import numpy as np
import pytest

from tests import datagen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k", [(129, 132, 300), (1, 128, 1), (255, 256, 257), (4097, 200, 1025), (20_000, 1024, 2_100), (12_345, 384, 5_000)])
@pytest.mark.parametrize("lists", [3, 4, 5, 9], ids=["none", "roomy", "overflowing", "dropping"])
def test_tensor_core_routes_agree_with_the_simt_search(n, d, k, lists):
    import superkmeans_b200 as skm

    eng = skm.engine
    if not eng.tensor_cores_enabled():
        pytest.skip("tensor cores are switched off")
    rng = np.random.default_rng(n)
    x = datagen.gaussian_mixture(n, d, max(1, k // 2), 0.3, k)
    y = x[rng.choice(n, k, replace=k > n)] + np.float32(0.02) * rng.standard_normal((k, d), dtype=np.float32)
    prev, _ = eng.find_nearest(x, y)
    far = rng.random(n) < 0.2
    prev[far] = rng.integers(0, k, far.sum())
    vd = eng.dimension_split(d)[1]
    for pd in sorted({min(16, vd), min(vd, 17 + vd // 2), vd}):   # one slice of 16, a ragged one, all of them
        try:
            eng.set_prune_split(1)
            want, want_dist, want_kept = eng.find_nearest_pruned(x, y, prev, pd)
            eng.set_prune_split(lists)
            knn, dist, kept = eng.find_nearest_pruned(x, y, prev, pd)
        finally:
            eng.set_prune_split(0)
        assert (knn != want).sum() <= n // 2000
        same = knn == want
        assert np.abs(dist - want_dist)[same].max() <= 1e-5 * max(1.0, float(want_dist.max()))
        assert np.abs(kept.astype(np.int64) - want_kept.astype(np.int64)).sum() <= 2 + 5e-3 * want_kept.sum()


@pytest.mark.parametrize("lists", [4, 9], ids=["roomy", "dropping"])
@pytest.mark.parametrize("kind", ["outlier 1e4", "outlier 1e7", "outlier 1e10", "outlier 1e18", "infinite outlier", "spread", "small", "zero"])
def test_centroids_of_very_different_norms(kind, lists):
    import superkmeans_b200 as skm

    eng = skm.engine
    if not eng.tensor_cores_enabled():
        pytest.skip("tensor cores are switched off")
    n, d, k = 6_000, 512, 700
    rng = np.random.default_rng(len(kind))
    x = datagen.gaussian_mixture(n, d, k // 2, 0.3, 9)
    y = x[rng.choice(n, k, replace=False)] + np.float32(0.02) * rng.standard_normal((k, d), dtype=np.float32)
    if kind.startswith("outlier"):
        y[k // 3] *= np.float32(kind.split()[1])
    elif kind == "infinite outlier":
        y[k // 3, 7] = np.inf
    elif kind == "spread":      # points and centroids of all sizes
        s = (10.0 ** rng.uniform(-6, 6, (n, 1))).astype(np.float32)
        x, y = x * s, y * (10.0 ** rng.uniform(-6, 6, (k, 1))).astype(np.float32)
    elif kind == "small":       # squared norms at the lower end of fp32
        x, y = x * np.float32(4e-19), y * np.float32(4e-19)
    else:
        y[k // 3] = 0
    # the previous centroid: the nearest, or, for a third of the points, the one after it (further ones overflow the lists)
    xd, yd = x.astype(np.float64), np.where(np.isfinite(y), y, np.float32(1e18)).astype(np.float64)
    order = np.argpartition((yd ** 2).sum(1)[None, :] - 2 * xd @ yd.T, 1, axis=1)[:, :2].astype(np.uint32)
    two = np.stack([((xd - yd[order[:, i]]) ** 2).sum(1) for i in range(2)], 1).argsort(1)
    prev = order[np.arange(n), two[np.arange(n), (rng.random(n) < 0.33).astype(int)]]
    for pd in (16, 100, eng.dimension_split(d)[1]):
        try:
            eng.set_prune_split(1)
            want, want_dist, want_kept = eng.find_nearest_pruned(x, y, prev, pd)
            eng.set_prune_split(lists)
            knn, dist, kept = eng.find_nearest_pruned(x, y, prev, pd)
        finally:
            eng.set_prune_split(0)
        assert (knn != want).sum() <= n // 1000, (pd, (knn != want).sum())
        same = knn == want
        scale = (x.astype(np.float64) ** 2).sum(1)[same] + want_dist[same]
        # the fp32 search sums a distance by differences, the listed one recomputes it so: a rounding per sum of 64
        assert (np.abs(dist.astype(np.float64) - want_dist)[same] <= 1e-5 * scale).all()
        assert np.abs(kept.astype(np.int64) - want_kept.astype(np.int64)).sum() <= 2 + 5e-3 * want_kept.sum(), (pd, kept.sum(), want_kept.sum())


# squared norms below the smallest normal float, and within a tenth of the largest
@pytest.mark.parametrize("length", [1e-20, 3e-21, 1.75e19, 1.83e19])
def test_rows_at_the_ends_of_what_floats_hold(length):
    """Every row has a previous centroid near it, which leaves few to look at, and a nearer one."""
    from superkmeans_b200 import engine

    n, k, d = 900, 300, 256
    rng = np.random.default_rng(3)
    y = np.empty((2 * k, d))
    y[0::2] = rng.standard_normal((k, d))
    y[1::2] = y[0::2] + 0.5 * rng.standard_normal((k, d))
    at = 2 * rng.integers(0, k, n)
    x = y[at] + 0.1 * rng.standard_normal((n, d))
    scale = length / np.linalg.norm(np.concatenate([x, y]), axis=1).max()
    x, y, prev = (x * scale).astype(np.float32), (y * scale).astype(np.float32), (at + 1).astype(np.uint32)
    for mode in (1, 4):
        engine.set_prune_split(mode)
        try:
            knn = engine.find_nearest_pruned(x, y, prev, 96)[0]
        finally:
            engine.set_prune_split(0)
        assert (knn == at).mean() >= 0.99, (mode, (knn == at).mean())   # the search may drop a centroid on the way
