"""Column tiles that centroids fill in part, without groups and with them, and assignments that ask for no distances."""
import numpy as np
import pytest

from tests import datagen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k", [(120_000, 256, k) for k in (1, 2, 15, 16, 17, 31, 33, 127, 129, 255, 256, 257, 273)] + [(20_000, 384, 4_100), (30_001, 1_536, 2_500), (19_200, 1_028, 3_000),
                                                                                                                        (20_003, 50, 2_500), (20_000, 1_024, 3_001)])
def test_assignments_with_and_without_distances(n, d, k):
    import torch

    import superkmeans_b200 as skm

    g = torch.Generator(device="cuda").manual_seed(n + d + k)
    c = torch.randn(k, d, generator=g, device="cuda")
    x = c[torch.randint(k, (n,), generator=g, device="cuda")] + 0.5 * torch.randn(n, d, generator=g, device="cuda")
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    skm.Engine(k, d).assign(x, c, n=n, on_device=True, out=out)
    knn, _ = skm.engine.find_nearest(x.cpu().numpy(), c.cpu().numpy())
    assert out.min() >= 0 and out.max() < k
    norms = (x.double() ** 2).sum(1) + (c.double() ** 2).sum(1).max()
    for a in (out.long(), torch.from_numpy(knn.astype(np.int64)).cuda()):
        for rows in torch.arange(n, device="cuda").split(8192):
            true = torch.cdist(x[rows].double(), c.double()) ** 2
            mine = true.gather(1, a[rows][:, None])[:, 0]
            assert ((mine - true.min(1).values) <= 1e-6 * norms[rows]).all()    # fp32 sums of d products


@pytest.mark.parametrize("n,d,k", [(20_000, 96, 64), (60_000, 64, 1_000), (80_000, 128, 4_300), (150_000, 32, 66_000)])
def test_groups_of_many_sizes(n, d, k):
    """Fine clusterings of 8, some 30, some 65 and some 257 centroids; the sequential form assigns each of them by itself."""
    import superkmeans_b200 as skm

    x = datagen.gaussian_mixture(n, d, max(8, k // 3), 0.3, n)
    res = []
    for trace in (True, False):
        e = skm.Engine(k, d, skm.default_config(True, early_termination=0, suppress_warnings=1, iters_fineclustering=1), hierarchical=True)
        e.set_trace(trace)
        e.train(x)
        res.append((e.assignments(), np.array([s.objective for s in e.stats(2)])))
    (a0, o0), (a1, o1) = res
    assert len(o0) == len(o1) and np.abs(o0 - o1).max() <= 1e-5 * max(float(o0.max()), 1e-12)   # distances near zero carry the rounding of the norms
    assert (a0 == a1).mean() >= 0.99
