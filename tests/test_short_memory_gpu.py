"""Steps that need more memory than the way they replaced take that way when the memory is not there (a test hook makes the
allocations of some sizes fail)."""
import contextlib

import numpy as np
import pytest

from tests import datagen

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def without(least, most=None, pinned=False):
    from superkmeans_b200 import _lib

    _lib.lib.skm_debug_alloc_failures(least, least if most is None else most, int(pinned))
    try:
        yield
    finally:
        _lib.lib.skm_debug_alloc_failures(1, 0, int(pinned))


@pytest.mark.parametrize("beside", [False, True], ids=["asked for", "beside a training"])
@pytest.mark.parametrize("pinned", [False, True])
def test_rotation_matrix(pinned, beside):
    import superkmeans_b200 as skm

    d, n = 500, 400
    # the scratch has four matrices of 512 x 512 doubles, the draws on the host at least d x d floats of pinned memory
    with without(*((4 * d * d, 1 << 40, True) if pinned else (8 * 512 * 512, 8 * 512 * 512, False))):
        e = skm.Engine(4, d, skm.default_config(False, sampling_fraction=1.0, iters=2))
        if beside:
            x = np.random.default_rng(0).standard_normal((n, d), dtype=np.float32)
            assert np.isfinite(e.train(x)).all()
        m = e.get_rotation()
    np.testing.assert_array_equal(m, skm.engine.rotation_matrix(d, 42))


def test_rotation_of_odd_rows():
    from superkmeans_b200 import engine

    n, d = 20_000, 130
    rng = np.random.default_rng(0)
    x, m = rng.standard_normal((n, d), dtype=np.float32), rng.standard_normal((d, d), dtype=np.float32)
    with without(4 * n * (d + 2), 4 * n * (d + 2) + 16 * d * (d + 6)):   # the padded rows and the halves of the matrix
        got = engine.rotate(m, x, to_assign=True)
    np.testing.assert_array_equal(got, engine.rotate(m, x))   # the fp32 tiles


def test_list_route():
    import superkmeans_b200 as skm

    n, d, k = 20_000, 256, 400
    vertical = skm.engine.dimension_split(d)[1]
    x = datagen.gaussian_mixture(n, d, k, 0.3, 4)

    def train():
        e = skm.Engine(k, d, skm.default_config(False, sampling_fraction=1.0, iters=5, early_termination=0))
        e.train(x)
        return e.assignments(), e.last_prune_path

    want, path = train()
    assert path == 4
    with without(2 * n * vertical):   # a half of all points' leading columns
        got, path = train()
    assert path == 6
    assert (got == want).mean() >= 0.999


def test_dense_chain_of_a_training():
    """Unstructured rows go through the dense chain from the first pruned pass on."""
    import superkmeans_b200 as skm

    n, d, k = 20_000, 256, 400
    x = np.random.default_rng(0).standard_normal((n, d), dtype=np.float32)

    def train():
        e = skm.Engine(k, d, skm.default_config(False, sampling_fraction=1.0, iters=3, early_termination=0, data_already_rotated=1))
        c = e.train(x)
        return c, e.assignments(), e.last_prune_path

    want = train()
    assert want[2] == 3
    with without(4 * n * d + 1, 4 * n * (d + 128)):   # the halves of all points, whose segments are padded to 64 columns
        got = train()
    for a, b in zip(want, got):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("least", [4_900, 2_500, 1_000])
def test_dense_chain(least):
    from superkmeans_b200 import _lib, engine

    n, d, k = 20_000, 256, 400
    x = datagen.gaussian_mixture(n, d, k, 0.3, 4)
    y = datagen.gaussian_mixture(k, d, k, 0.3, 5)
    prev = np.random.default_rng(0).integers(0, k, n).astype(np.uint32)
    pitch = 320   # d' = 96: segments of 96, 64 and 96 columns
    engine.set_prune_split(3)
    try:
        want = engine.find_nearest_pruned(x, y, prev, 96)
        _lib.lib.skm_debug_chain_slice(9_728)
        with without(4 * least * pitch, 4 * 9_728 * pitch):
            got = engine.find_nearest_pruned(x, y, prev, 96)
    finally:
        _lib.lib.skm_debug_chain_slice(0)
        engine.set_prune_split(0)
    for a, b in zip(want, got):
        np.testing.assert_array_equal(a, b)


def test_exact_assignment():
    import torch

    import superkmeans_b200 as skm

    n, d, k = 20_000, 96, 2_000
    x = datagen.gaussian_mixture(n, d, k, 0.3, 4)
    c = x[:k].copy()
    xd, cd, out = torch.from_numpy(x).cuda(), torch.from_numpy(c).cuda(), torch.empty(n, dtype=torch.int32, device="cuda")

    def answers():
        e = skm.Engine(k, d)
        e.assign(xd, cd, n=n, on_device=True, out=out)
        t = skm.Engine(k, d, skm.default_config(False, sampling_fraction=1.0, iters=1, early_termination=0))
        t.train(x)
        return [skm.engine.find_nearest(x, c)[0], e.assign(x, c), out.cpu().numpy().view(np.uint32), t.assignments()]

    want = answers()
    launches = skm.engine.kernel_launches()
    with without(2 * n * d):   # the fp16 rows of the filter
        got = answers()
    assert skm.engine.kernel_launches() > launches
    for a, b in zip(want, got):
        assert (a != b).sum() <= 2   # rows at the same distance from two centroids
    # a third of the rows has more equally near centroids than the filter keeps and is decided, slice after slice
    x[::3], c[k // 2:] = x[0], x[0]
    want = skm.engine.find_nearest(x, c)[0]
    with without(12 * n * d // 10, 15 * n * d // 10):
        np.testing.assert_array_equal(skm.engine.find_nearest(x, c)[0], want)


def test_fine_clusterings():
    import superkmeans_b200 as skm

    n, d, k = 20_000, 96, 200
    x = datagen.gaussian_mixture(n, d, k // 3, 0.3, 4)

    def train():
        e = skm.Engine(k, d, skm.default_config(True, early_termination=0, suppress_warnings=1), hierarchical=True)
        e.train(x)
        return e.assignments(), [(s.iteration, s.objective) for s in e.stats(2)]

    want, stats = train()
    with without(2 * n * d):   # the fp16 rows of all mesoclusters
        got, again = train()
    assert [i for i, _ in stats] == [i for i, _ in again]
    assert (got == want).mean() >= 0.98
    # the first pass of every mesocluster starts from the same rows
    a, b = (np.array([o for i, o in s if i == 1]) for s in (stats, again))
    assert np.abs(a - b).max() <= 1e-5 * a.max()
