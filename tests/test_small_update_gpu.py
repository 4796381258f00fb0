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


@pytest.mark.parametrize("n,d", [(512, 1_024), (2_048, 256), (8_192, 64)])
def test_sums_of_many_equal_rows(n, d):
    """512 rows a thread, of values that a sum of more than 256 of them rounds off all in one direction."""
    import superkmeans_b200 as skm

    v = (1.0 + np.linspace(0.5, 1.0, d) * 2.0 ** -16).astype(np.float32)
    e = skm.Engine(1, d, skm.default_config(False, iters=1, sampling_fraction=1.0, early_termination=0, data_already_rotated=1))
    e.set_trace(True)
    e.train(np.tile(v, (n, 1)))
    # half a unit of every partial sum: 2^-24 (1 + .. + 128) / 128 in a chain of 128 rows, and as in a chain of 32 for what adds such sums up
    error = np.abs(e.trace()[-1]["centroids"][0].astype(np.float64) / v - 1)
    assert error.max() <= 2.0 ** -24 * (129 / 2 + 33 / 2 + 1), error.max()
