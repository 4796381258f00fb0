"""The dense chain on the tensor cores against the one in fp32, at the edges of its tiles (256 points, units of 256 centroids, chunks of
1024) and of its segments."""
import numpy as np
import pytest

from tests import datagen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,d", [(1, 300, 132), (127, 257, 132), (129, 1_025, 200), (256, 1_024, 128), (257, 256, 260), (4_608, 1_300, 384), (4_609, 2_049, 256), (20_000, 513, 1_000),
                                   (700, 5, 768), (700, 3_000, 1_540)])
def test_chain_on_the_tensor_cores(n, k, d):
    from superkmeans_b200 import engine

    x = datagen.gaussian_mixture(n, d, max(k // 4, 1), 0.4, n + k)
    y = datagen.gaussian_mixture(k, d, max(k // 4, 1), 0.4, k)
    # rows of different magnitudes: every row has a scale of its own
    x *= (10.0 ** np.random.default_rng(n).uniform(-3, 3, (n, 1))).astype(np.float32)
    prev = np.random.default_rng(d).integers(0, k, n).astype(np.uint32)
    vertical = engine.dimension_split(d)[1]
    for partial in {16, vertical // 2, vertical - 3, vertical}:
        out = {}
        for mode in (2, 3):
            engine.set_prune_split(mode)
            try:
                out[mode] = engine.find_nearest_pruned(x, y, prev, partial)
            finally:
                engine.set_prune_split(0)
        knn, dist = out[3][0], out[3][1]
        exact = ((x.astype(np.float64) - y[knn].astype(np.float64)) ** 2).sum(1)
        assert (np.abs(dist - exact) <= 1e-5 * exact + 1e-12).all()
        # pairs within rounding of a threshold of the search
        assert (knn == out[2][0]).mean() >= 0.999 - 1.0 / n
        assert abs(float(out[3][2].sum()) - float(out[2][2].sum())) <= 1e-3 * float(out[2][2].sum()) + 2


@pytest.mark.parametrize("n,d", [(500, 132), (700, 256), (500, 768), (1_200, 1_024), (500, 1_536), (5_000, 384)])
def test_a_centroid_a_little_nearer_than_the_previous_one(n, d):
    """Every row has its previous centroid and one that is nearer by less than the rounding of the tensor cores' sums: the refinement sees it,
    whatever those sums say."""
    from superkmeans_b200 import engine

    rng = np.random.default_rng(d)
    x = rng.standard_normal((n, d))
    x /= np.linalg.norm(x, axis=1, keepdims=True)

    def away(r):
        u = rng.standard_normal((n, d))
        return x + r * u / np.linalg.norm(u, axis=1, keepdims=True)

    y = np.empty((2 * n, d))
    y[0::2], y[1::2] = away(0.3), away(0.3 * (1 - 5e-6))
    x, y, prev = x.astype(np.float32), y.astype(np.float32), np.arange(0, 2 * n, 2, dtype=np.uint32)
    found = {}
    for mode in (2, 3):
        engine.set_prune_split(mode)
        try:
            found[mode] = engine.find_nearest_pruned(x, y, prev, engine.dimension_split(d)[1] // 2)[0] == prev + 1
        finally:
            engine.set_prune_split(0)
    # the search may drop it on the way, in either form; what the fp32 form finds is found, but for pairs within rounding of a threshold
    assert found[2].mean() >= 0.5
    assert (found[3] | ~found[2]).mean() >= 0.99, (found[2].mean(), found[3].mean())


# squared norms below the smallest normal float, and within a tenth of the largest
@pytest.mark.parametrize("length", [1e-20, 3e-21, 1.75e19, 1.83e19])
def test_rows_at_the_ends_of_what_floats_hold(length):
    from superkmeans_b200 import engine

    n, k, d = 700, 300, 256
    rng = np.random.default_rng(7)
    y = rng.standard_normal((k, d))
    y /= np.linalg.norm(y, axis=1, keepdims=True)
    at = rng.integers(0, k, n)
    x = y[at] + 0.3 / np.sqrt(d) * rng.standard_normal((n, d))
    x /= np.linalg.norm(x, axis=1, keepdims=True)
    x, y, prev = (x * length).astype(np.float32), (y * length).astype(np.float32), rng.integers(0, k, n).astype(np.uint32)
    for mode in (2, 3):
        engine.set_prune_split(mode)
        try:
            knn = engine.find_nearest_pruned(x, y, prev, 96)[0]
        finally:
            engine.set_prune_split(0)
        assert (knn == at).mean() >= 0.99, (mode, (knn == at).mean())   # the search may drop a centroid on the way
