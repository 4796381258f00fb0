"""Lists of nearest rows behind the recall of a Train, for list lengths and row counts around a round of 256 rows, a full buffer and a
slab of 16 384 rows: the recall of a first iteration against one computed from the returned centroids and assignments."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,objective_k,explore", [(300, 3, 300, 0.5), (2_000, 255, 1, 0.004), (2_100, 257, 700, 0.3), (20_000, 300, 100, 0.01), (34_000, 64, 1_536, 0.1)])
def test_recall_of_one_iteration(n, k, objective_k, explore):
    import superkmeans_b200 as skm

    d = 36
    rng = np.random.default_rng(n + k)
    x = rng.standard_normal((n, d), dtype=np.float32)
    q = rng.standard_normal((50, d), dtype=np.float32)
    e = skm.Engine(k, d, skm.default_config(False, iters=1, sampling_fraction=1.0, early_termination=0, objective_k=objective_k, ann_explore_fraction=explore, suppress_warnings=1,
                                            data_already_rotated=1, unrotate_centroids=0))
    c = e.train(x, queries=q)
    recall, visited = e.stats(0)[0].recall, max(1, int(k * explore))
    assign = e.assignments()
    x64, q64, c64 = x.astype(np.float64), q.astype(np.float64), c.astype(np.float64)

    def nearest(y, m):
        dist = (y ** 2).sum(1) - 2 * q64 @ y.T
        return np.argpartition(dist, min(m, len(y)) - 1, axis=1)[:, :m] if m < len(y) else np.tile(np.arange(len(y)), (len(q64), 1))

    near, clusters = nearest(x64, objective_k), nearest(c64, visited)
    hits = sum(np.isin(assign[near[i]], clusters[i]).sum() for i in range(len(q)))
    assert abs(recall - hits / near.size) <= 2.0 / near.size + 1e-3, (recall, hits / near.size)   # a pair of equally near rows or centroids
