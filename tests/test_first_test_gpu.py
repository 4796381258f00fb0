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
