"""Sums, means, costs and shifts of small problems, which one launch makes, at the borders of that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,d,skewed", [(64, 3, 32, False), (8_191, 17, 64, False), (8_192, 17, 64, True), (8_193, 17, 64, False), (512, 5, 1_024, False), (514, 5, 1_020, True),
                                          (4_096, 341, 128, False), (4_097, 341, 96, True), (4_096, 342, 128, False), (5_000, 100, 100, False), (16_384, 2, 32, True)])
def test_an_iteration_of_a_small_problem(n, k, d, skewed):
    import superkmeans_b200 as skm

    rng = np.random.default_rng(n + k + d)
    x = rng.standard_normal((n, d), dtype=np.float32)
    if skewed:   # all but a few in one place
        x[k * 2:] = x[0] + np.float32(1e-3) * x[k * 2:]
    e = skm.Engine(k, d, skm.default_config(False, iters=3, sampling_fraction=1.0, early_termination=0, data_already_rotated=1))
    e.set_trace(True)
    c = e.train(x)
    before = None
    for i, (snap, st) in enumerate(zip(e.trace(), e.stats())):
        a, dist = snap["assign"], snap["dist"]
        counts = np.bincount(a, minlength=k)
        np.testing.assert_array_equal(counts, snap["sizes_pre"])
        assert abs(st.objective - dist.astype(np.float64).sum()) <= 1e-6 * dist.astype(np.float64).sum()
        means = np.zeros((k, d))
        np.add.at(means, a, x.astype(np.float64))
        means /= np.maximum(counts, 1)[:, None]
        if st.split == 0:
            # 32-bit sums of at most n terms in eight or more chains
            assert np.abs(snap["centroids"] - means).max() <= 1e-7 * n / 8 * np.abs(x).max() + 1e-6
            if before is not None:
                want = ((snap["centroids"].astype(np.float64) - before) ** 2).sum()
                assert abs(st.shift - want) <= 1e-4 * want + 1e-9
        before = snap["centroids"].astype(np.float64)
    np.testing.assert_array_equal(c, e.trace()[-1]["centroids"])
