"""Centroid sums at the sizes where the sort's units and the segmented sum's tiles change."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,d", [(1, 1, 1), (127, 5, 3), (128, 5, 4), (129, 40, 64), (2047, 256, 130), (6000, 91, 768), (131071, 300, 20), (131072, 300, 20),
                                   (151551, 77, 12), (151552, 77, 12), (1048575, 5, 4), (1048576, 5, 4), (5000, 257, 8), (5000, 1024, 8), (5000, 1025, 8), (300_000, 1000, 8)])
def test_update_centroids_at_the_edges(n, k, d):
    import superkmeans_b200 as skm

    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, d), dtype=np.float32)
    a = rng.integers(0, k, n).astype(np.uint32)
    dist = rng.random(n, dtype=np.float32)
    sums, counts, wcss = skm.engine.update_centroids(x, a, k, dist)
    expected = np.zeros((k, d))
    np.add.at(expected, a, x.astype(np.float64))
    np.testing.assert_array_equal(counts, np.bincount(a, minlength=k))
    assert np.abs(sums - expected).max() <= 1e-5 * max(1.0, np.abs(expected).max())
    assert abs(wcss - dist.astype(np.float64).sum()) <= 1e-6 * max(1.0, wcss)
    np.testing.assert_array_equal(sums, skm.engine.update_centroids(x, a, k, dist)[0])
