"""Exact assignment at sizes around the borders of its three ways (direct, filter, blocks) and of their tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(n, k, d, kind, seed):
    rng = np.random.default_rng(seed)
    c = rng.standard_normal((k, d), dtype=np.float32)
    x = c[rng.integers(0, k, n)] + np.float32(0.5) * rng.standard_normal((n, d), dtype=np.float32)
    if kind == "offset":          # norms far above the spread
        x, c = x + np.float32(10), c + np.float32(10)
    elif kind == "twins":         # every centroid twice: the lower index wins
        c[k // 2:] = c[:k - k // 2]
    elif kind == "scales":        # rows of very different norms
        x *= 10.0 ** rng.uniform(-4, 4, (n, 1)).astype(np.float32)
    elif kind == "tiny":          # squared norms below the filter's range
        x, c = x * np.float32(1e-18), c * np.float32(1e-18)
    elif kind == "same":          # more equally near centroids than the filter keeps
        x[:], c[:] = x[0], c[0]
    elif kind == "zero":
        x[::3], c[::5] = 0, 0
    return x, c


@pytest.mark.parametrize("n,k,d,kind", [
    (1, 1, 1, ""), (1, 1000, 768, ""), (3, 77, 33, ""), (8, 5000, 384, ""), (9, 65, 17, ""), (64, 64, 16, ""), (65, 129, 64, ""), (5, 70_000, 16, ""),   # direct
    (20_001, 2_500, 50, ""), (10_000, 2_777, 33, ""), (30_000, 4_096, 384, ""), (9_001, 2_049, 1_536, ""), (19_200, 3_000, 768, ""), (40_000, 1_025, 7, ""),   # filter
    (120_000, 40, 256, ""),   # blocks
    (20_000, 2_000, 96, "offset"), (20_000, 2_000, 96, "twins"), (20_000, 2_000, 96, "scales"), (20_000, 2_000, 96, "tiny"), (20_000, 2_000, 96, "same"),
    (20_000, 2_000, 96, "zero"), (20_000, 2_000, 95, "twins")])
def test_nearest_centroid_on_every_route(n, k, d, kind):
    import torch

    import superkmeans_b200 as skm

    x, c = _data(n, k, d, kind, n + k + d)
    knn, dist = skm.engine.find_nearest(x, c)
    assert knn.max() < k
    a = torch.from_numpy(knn.astype(np.int64)).cuda()
    xd, cd, dd = torch.from_numpy(x).cuda().double(), torch.from_numpy(c).cuda().double(), torch.from_numpy(dist).cuda().double()
    scale_c = (cd ** 2).sum(1).max()
    for rows in torch.arange(n, device="cuda").split(4096):
        true = torch.cdist(xd[rows], cd) ** 2
        mine = true.gather(1, a[rows][:, None])[:, 0]
        scale = (xd[rows] ** 2).sum(1) + scale_c
        assert ((mine - true.min(1).values) <= 1e-6 * scale).all()
        assert ((dd[rows] - mine).abs() <= 2e-6 * scale).all()
    if kind == "twins":
        assert (knn < k - k // 2).all()
