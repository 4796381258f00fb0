"""Rotation GEMM at the edges of its tiles (256 rows and columns, 32 columns of K per stage, four parts of K)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d", [(1, 32), (129, 36), (257, 64), (600, 80), (400, 176), (255, 256), (513, 260), (300, 772), (38_000, 300), (777, 1_536)])
def test_rotation_and_back(n, d):
    import superkmeans_b200 as skm

    rng = np.random.default_rng(n + d)
    x = rng.standard_normal((n, d), dtype=np.float32)
    m = rng.standard_normal((d, d), dtype=np.float32)
    scale = np.linalg.norm(x.astype(np.float64), axis=1)[:, None]
    for got, mat in ((skm.engine.rotate(m, x), m.T), (skm.engine.rotate(m, x, to_assign=True), m.T), (skm.engine.unrotate(m, x), m)):
        want = x.astype(np.float64) @ mat.astype(np.float64)
        assert (np.abs(got - want) <= 3e-6 * scale * np.linalg.norm(mat.astype(np.float64), axis=0)).all()
