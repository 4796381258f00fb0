"""What happens when something inside a tensor-core kernel does not arrive.

Every wait inside those kernels is bounded.  The test below makes one run out in the allowed way: the TMA producer is
told to stop early (a test hook of the C ABI), so the other roles wait for tiles that nothing will ever deliver, the
shortened limit expires, the kernel records a code and returns, and the call reports an error.  Nothing faults or hangs;
the same process then runs the same operator normally."""
import numpy as np
import pytest

from tests import datagen

pytestmark = pytest.mark.gpu


def test_a_wait_that_runs_out_is_reported_and_leaves_the_context_usable():
    from superkmeans_b200 import _lib, engine

    if not engine.tensor_cores_enabled():
        pytest.skip("the tensor-core kernels are switched off")
    n, d, k = 4096, 256, 700
    x = datagen.gaussian_mixture(n, d, k, 0.3, 3)
    y = x[:k].copy()
    want, _ = engine.find_nearest(x, y)
    # about a tenth of a second at 2 GHz; the producer stops after three of the 16 k-blocks of the first tile
    _lib.check(_lib.lib.skm_debug_wait_injection(200_000_000, 3))
    try:
        with pytest.raises(RuntimeError, match="gave up waiting on a barrier"):
            engine.find_nearest(x, y)
    finally:
        _lib.check(_lib.lib.skm_debug_wait_injection(0, 0))
    got, dist = engine.find_nearest(x, y)
    np.testing.assert_array_equal(got, want)
    assert (dist >= 0).all()


@pytest.fixture
def early_stop():
    """Producers that stop after one stage, waits of a tenth of a second."""
    from superkmeans_b200 import _lib, engine

    if not engine.tensor_cores_enabled():
        pytest.skip("the tensor-core kernels are switched off")

    class Stop:
        def __enter__(self):
            _lib.check(_lib.lib.skm_debug_wait_injection(200_000_000, 1))

        def __exit__(self, *_):
            _lib.check(_lib.lib.skm_debug_wait_injection(0, 0))
            engine.set_prune_split(0)

    yield Stop()
    _lib.check(_lib.lib.skm_debug_wait_injection(0, 0))
    engine.set_prune_split(0)


@pytest.mark.parametrize("n,k,d", [(120_000, 40, 256), (12_000, 2_048, 384)], ids=["three products", "filter"])
def test_exact_assignment(early_stop, n, k, d):
    from superkmeans_b200 import engine

    x = datagen.gaussian_mixture(n, d, k, 0.3, 3)
    y = x[:k].copy()
    want, _ = engine.find_nearest(x, y)
    with early_stop, pytest.raises(RuntimeError, match="gave up waiting on a barrier"):
        engine.find_nearest(x, y)
    np.testing.assert_array_equal(engine.find_nearest(x, y)[0], want)


@pytest.mark.parametrize("which", ["of a training", "to assign", "back"])
def test_rotation(early_stop, which):
    from superkmeans_b200 import engine

    rng = np.random.default_rng(1)
    x, m = rng.standard_normal((3_000, 256), dtype=np.float32), rng.standard_normal((256, 256), dtype=np.float32)

    def rotate():
        return engine.unrotate(m, x) if which == "back" else engine.rotate(m, x, to_assign=which == "to assign")

    want = rotate()
    with early_stop, pytest.raises(RuntimeError, match="gave up waiting on a barrier"):
        rotate()
    np.testing.assert_array_equal(rotate(), want)


@pytest.mark.parametrize("n,mode", [(4_096, 4), (4_096, 9), (2_000, 3), (30_000, 3)], ids=["first test", "first test that drops", "chain in slices", "chain"])
def test_pruned_search(early_stop, n, mode):
    from superkmeans_b200 import engine

    d, k = 256, 1_500
    x = datagen.gaussian_mixture(n, d, k, 0.3, 3)
    y = x[:k].copy() if n >= k else np.concatenate([x, x])[:k].copy()
    prev, _ = engine.find_nearest(x, y)
    prev = np.where(np.arange(n) % 3 == 0, (prev + 1) % k, prev)
    engine.set_prune_split(mode)
    want = engine.find_nearest_pruned(x, y, prev, 48)
    with early_stop, pytest.raises(RuntimeError, match="gave up waiting on a barrier"):
        engine.find_nearest_pruned(x, y, prev, 48)
    engine.set_prune_split(mode)
    got = engine.find_nearest_pruned(x, y, prev, 48)
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("where", ["host", "device"])
@pytest.mark.parametrize("fraction", [1.0, 0.9])
def test_assignment_of_training_points(early_stop, where, fraction):
    import torch

    import superkmeans_b200 as skm

    n, d, k = 20_000, 256, 400
    x = datagen.gaussian_mixture(n, d, k, 0.3, 3)
    # rows that are rotated already: the first kernel with waits is the first test
    e = skm.Engine(k, d, skm.default_config(False, iters=3, sampling_fraction=fraction, max_points_per_cluster=1000, early_termination=0, data_already_rotated=1))
    c = e.train(x)

    def call():
        if where == "host":
            return e.assign_training_points(x, c)
        out = torch.empty(n, dtype=torch.int32, device="cuda")
        e.assign_training_points(torch.from_numpy(x).cuda(), torch.from_numpy(c).cuda(), n=n, on_device=True, out=out)
        return out.cpu().numpy().view(np.uint32)

    with early_stop, pytest.raises(RuntimeError, match="gave up waiting on a barrier"):
        call()
    # the next call is about itself alone
    a = e.assign(x, c)
    got = call()
    assert (got == a).mean() >= 0.995


@pytest.mark.parametrize("hierarchical", [False, True])
def test_training(early_stop, hierarchical):
    import superkmeans_b200 as skm

    n, d, k = 20_000, 256, 400
    x = datagen.gaussian_mixture(n, d, k, 0.3, 3)

    def train():
        e = skm.Engine(k, d, skm.default_config(hierarchical, early_termination=0, suppress_warnings=1), hierarchical=hierarchical)
        return e.train(x)

    want = train()
    with early_stop, pytest.raises(RuntimeError, match="gave up waiting on a barrier"):
        train()
    np.testing.assert_allclose(train(), want, atol=1e-3)
