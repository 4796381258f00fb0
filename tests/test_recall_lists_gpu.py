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


# after seven rounds of 256 rows the buffer of 2048 keys is one key short of a flush
@pytest.mark.parametrize("n,objective_k", [(1_792, 5), (1_793, 5), (2_048, 5), (2_304, 256), (2_304, 300), (6_000, 1_536)])
def test_lists_of_many_queries_repeat_themselves(n, objective_k):
    """A list is full, or not, for all warps of its block at once: thousands of lists, several times over, give one recall."""
    import superkmeans_b200 as skm

    d, k = 32, 40
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, d), dtype=np.float32)
    q = rng.standard_normal((3_000, d), dtype=np.float32)
    recalls = set()
    for _ in range(5):
        e = skm.Engine(k, d, skm.default_config(False, iters=2, sampling_fraction=1.0, early_termination=0, objective_k=objective_k, ann_explore_fraction=0.1, suppress_warnings=1,
                                                data_already_rotated=1, unrotate_centroids=0))
        c = e.train(x, queries=q)
        recalls.add(tuple(s.recall for s in e.stats(0)))
    assert len(recalls) == 1
    assign = e.assignments()
    q64 = q.astype(np.float64)
    # (the recall of an iteration looks at the centroids that it ends with)
    rows = np.argpartition((x.astype(np.float64) ** 2).sum(1) - 2 * q64 @ x.astype(np.float64).T, objective_k - 1, axis=1)[:, :objective_k]
    clusters = np.argpartition((c.astype(np.float64) ** 2).sum(1) - 2 * q64 @ c.astype(np.float64).T, 3, axis=1)[:, :4]
    hits = sum(np.isin(assign[rows[i]], clusters[i]).sum() for i in range(len(q)))
    assert abs(recalls.pop()[-1] - hits / rows.size) <= 1e-3   # pairs of equally near rows or centroids
