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


def _centroids_in_vain(x, k, kind, rng):
    """Centroids that the filter cannot tell apart, so that it lists (nearly) every row, or those after the first ones."""
    c = x[rng.choice(len(x), k, replace=False)].copy()
    if kind == "outlier":
        c[k // 3] *= np.float32(1e6)
    elif kind == "nan":
        c[k // 3, 1] = np.nan
    elif kind == "copies":
        c = c[np.arange(k) % (k // 8)]
    elif kind == "later":      # the rows behind the first wave meet eight copies of their centroid
        c[k // 2:] = c[k // 2 + np.arange(k - k // 2) % (k // 16)]
        x[19_000:] = c[k // 2 + rng.integers(0, k // 16, len(x) - 19_000)] + np.float32(0.01) * rng.standard_normal((len(x) - 19_000, x.shape[1]), dtype=np.float32)
    elif kind == "earlier":    # only the rows of the first wave do
        c[k // 2:] = c[k // 2 + np.arange(k - k // 2) % (k // 16)]
        x[:19_000] = c[k // 2 + rng.integers(0, k // 16, 19_000)]
        x[19_000:] = c[rng.integers(0, k // 2, len(x) - 19_000)] + np.float32(0.01) * rng.standard_normal((len(x) - 19_000, x.shape[1]), dtype=np.float32)
    return c


@pytest.mark.parametrize("n,k,d", [(140_001, 16_384, 256), (120_000, 33_000, 50), (60_001, 2_048, 192)])
@pytest.mark.parametrize("kind", ["outlier", "nan", "copies", "later", "earlier"])
def test_rows_that_the_filter_cannot_settle(n, k, d, kind):
    import torch

    import superkmeans_b200 as skm

    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, d), dtype=np.float32)
    c = _centroids_in_vain(x, k, kind, rng)
    e = skm.Engine(k, d)
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    xd, cd = torch.from_numpy(x).cuda(), torch.from_numpy(c).cuda()
    e.assign(xd, cd, n=n, on_device=True, out=out)
    knn, dist = skm.engine.find_nearest(x, c)
    host = e.assign(x, c)
    y = torch.nan_to_num(cd, nan=1e18).double()   # a centroid that is no number is nobody's nearest
    scale_c = (torch.nan_to_num(cd, nan=0.0).double() ** 2).sum(1)
    for a in (out.cpu().numpy().view(np.uint32), knn, host):
        assert a.max() < k
        a = torch.from_numpy(a.astype(np.int64)).cuda()
        for rows in torch.arange(n, device="cuda").split(4096):
            true = torch.cdist(xd[rows].double(), y) ** 2
            mine = true.gather(1, a[rows][:, None])[:, 0]
            scale = (xd[rows].double() ** 2).sum(1) + scale_c[a[rows]]
            assert ((mine - true.min(1).values) <= 1e-6 * scale).all()
    assert np.isfinite(dist).all()


@pytest.mark.parametrize("kind", ["plain", "copies"])
def test_host_rows_that_the_filter_cannot_settle(kind):
    import torch

    import superkmeans_b200 as skm

    n, k, d = 280_000, 2_400, 256   # 287 MB: what the first piece came to decides about the others
    rng = np.random.default_rng(3)
    x = rng.standard_normal((n, d), dtype=np.float32)
    c = _centroids_in_vain(x, k, kind, rng)
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    xd, cd = torch.from_numpy(x).cuda(), torch.from_numpy(c).cuda()
    e = skm.Engine(k, d)
    e.assign(xd, cd, n=n, on_device=True, out=out)
    assert (e.assign(x, c) != out.cpu().numpy().view(np.uint32)).sum() <= 2
    t = skm.Engine(k, d, skm.default_config(False, sampling_fraction=1.0, iters=1, early_termination=0, data_already_rotated=0))
    t.train(x[:, :].copy())
    u = skm.Engine(k, d, skm.default_config(False, sampling_fraction=1.0, iters=1, early_termination=0))
    u.train(xd, n=n, on_device=True)
    assert (t.assignments() != u.assignments()).sum() <= 2
