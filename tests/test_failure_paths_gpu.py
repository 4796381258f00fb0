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


def test_rotation(early_stop):
    from superkmeans_b200 import engine

    rng = np.random.default_rng(1)
    x, m = rng.standard_normal((3_000, 256), dtype=np.float32), rng.standard_normal((256, 256), dtype=np.float32)
    want = engine.rotate(m, x)
    with early_stop, pytest.raises(RuntimeError, match="gave up waiting on a barrier"):
        engine.rotate(m, x)
    np.testing.assert_array_equal(engine.rotate(m, x), want)


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
