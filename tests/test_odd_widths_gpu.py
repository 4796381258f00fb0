"""Training on rows whose width is no multiple of four: the engine pads its own rows, which must not show."""
import numpy as np
import pytest

from tests import datagen

pytestmark = pytest.mark.gpu

WIDTHS = [33, 50, 130, 131, 133, 255]


@pytest.mark.parametrize("repeated", [False, True], ids=["distinct rows", "repeated rows"])
@pytest.mark.parametrize("d", WIDTHS)
def test_equals_the_restated_algorithm(d, repeated):
    import superkmeans_b200 as skm
    from oracle import restate

    n, k, iters, seed = 8_000, 300, 5, 3
    x = datagen.gaussian_mixture(n, d, k, 0.3, d)
    if repeated:   # equal first centroids: empty clusters, which are split off others with signs that alternate over the dimensions
        x[n // 2:] = x[:n - n // 2]
    m = skm.engine.rotation_matrix(d, seed)
    e = skm.Engine(k, d, skm.default_config(False, iters=iters, sampling_fraction=1.0, early_termination=0, seed=seed))
    e.set_rotation(m)
    np.testing.assert_array_equal(e.get_rotation(), m)
    c = e.train(x)
    want_c, want_rotated, want_a, stats = restate.train_flat(x, k, m, iters=iters, seed=seed)
    assert e.stats()[0].split == stats[0].split and e.stats()[1].partial_d == stats[1].partial_d
    assert (stats[0].split > 0) == repeated
    assert (e.assignments() == want_a).mean() >= 0.995
    # clusters with the same members: sums of 32-bit floats in another order
    same = np.array([np.array_equal(e.assignments() == i, want_a == i) for i in range(k)])
    assert same.mean() >= 0.9
    for got, want in ((c, want_c), (e.rotated_centroids(), want_rotated)):
        assert np.linalg.norm(got[same] - want[same], axis=1).max() <= 1e-4 * np.linalg.norm(want, axis=1).max()


@pytest.mark.parametrize("hierarchical,rotated,unrotate,angular", [(False, 1, 1, 0), (False, 0, 0, 0), (False, 0, 1, 1), (True, 0, 1, 0), (True, 1, 1, 0)])
@pytest.mark.parametrize("d", [51, 130, 257])
def test_centroids_are_means(d, hierarchical, rotated, unrotate, angular):
    import superkmeans_b200 as skm

    n, k = 30_000, 300
    x = datagen.gaussian_mixture(n, d, k, 0.3, d)
    cfg = skm.default_config(hierarchical, sampling_fraction=1.0, early_termination=0, data_already_rotated=rotated, unrotate_centroids=unrotate, angular=angular, suppress_warnings=1)
    e = skm.Engine(k, d, cfg, hierarchical=hierarchical)
    c = e.train(x)
    if not (rotated or unrotate):
        np.testing.assert_array_equal(c, e.rotated_centroids())
        c = c @ e.get_rotation()
    a = e.assignments()
    counts = np.bincount(a, minlength=k)
    means = np.zeros((k, d))
    np.add.at(means, a, x.astype(np.float64))
    means /= np.maximum(counts, 1)[:, None]
    if angular:
        means /= np.linalg.norm(means, axis=1, keepdims=True)
    # (the hierarchical form also draws clusters below a quarter of the average towards large ones)
    used = counts > (0.6 * n / k if hierarchical else 0)
    off = np.linalg.norm(c[used] - means[used], axis=1)
    assert np.median(off) <= 1e-5 and (off <= 2e-3).mean() >= 0.99   # (a split moves two centroids by a thousandth)
    if not hierarchical and not rotated and unrotate:
        again = e.assign_training_points(x, c)
        assert (again == e.assign(x, c)).mean() >= 0.98
