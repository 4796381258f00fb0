"""Centroids and rows with a NaN or an infinity: such a centroid is nobody's nearest, such a row has some answer, and the others
are what they are without them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,d", [(1, 300, 192), (2, 50, 7), (5, 300, 192), (8, 3_000, 50), (100, 40, 16), (3_169, 2_048, 192), (3_000, 70, 33), (5_000, 64, 64),   # direct
                                   (20_000, 2_000, 96), (20_000, 2_000, 95), (120_000, 40, 256)])   # filter, blocks
@pytest.mark.parametrize("value", [np.nan, -np.nan, np.inf, -np.inf])
def test_exact_assignment(n, k, d, value):
    import torch

    import superkmeans_b200 as skm

    rng = np.random.default_rng(n + k)
    x, c = rng.standard_normal((n, d), dtype=np.float32), rng.standard_normal((k, d), dtype=np.float32)
    want, want_dist = skm.engine.find_nearest(x, np.delete(c, [0, k // 3], axis=0))
    want = np.delete(np.arange(k), [0, k // 3])[want]
    c[[0, k // 3], d // 2] = value
    knn, dist = skm.engine.find_nearest(x, c)
    # (the products of the two calls are summed in different orders where the centroids' number changes the way)
    near = np.abs(dist - want_dist) <= 1e-5 * ((x.astype(np.float64) ** 2).sum(1) + d)
    assert near.all() and (knn != want).sum() <= n // 1000
    xd, cd = torch.from_numpy(x).cuda(), torch.from_numpy(c).cuda()
    if n <= 262_144:
        out, out_dist = torch.empty(n, dtype=torch.int32, device="cuda"), torch.empty(n, device="cuda")
        torch.cuda.synchronize()
        skm.engine.find_nearest_noalloc(xd.data_ptr(), cd.data_ptr(), n, k, d, out.data_ptr(), out_dist.data_ptr())
        assert (out.cpu().numpy() != want).sum() <= n // 1000
    # a row that is no number leaves the others alone
    x[n // 2, 0] = value
    again, dist = skm.engine.find_nearest(x, c)
    others = np.arange(n) != n // 2
    assert (again != knn)[others].sum() <= n // 1000 and again.max() < k and not np.isnan(dist).any()
