"""The rotation matrix made on the GPU against the host's (the same draws, the same factor, the same signs)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [42, 5])
@pytest.mark.parametrize("d", [1, 2, 31, 32, 33, 64, 65, 130, 200, 768, 1537])
def test_device_matrix_equals_the_host_one(d, seed):
    import superkmeans_b200 as skm

    host = skm.engine.rotation_matrix(d, seed)
    e = skm.Engine(4, d, skm.default_config(False, seed=seed))
    m = e.get_rotation()
    # both are rounded once from double, whose own error is 1e-7 of a rounding or less: at most a rounding apart, and in no more entries than
    # lie that close to the middle of two floats (at most 2 of a million were seen)
    assert np.abs(m - host).max() <= 1e-7
    assert (m != host).sum() <= 2 + 1e-5 * d * d
    assert np.abs(m.astype(np.float64) @ m.T.astype(np.float64) - np.eye(d)).max() <= 1e-6
