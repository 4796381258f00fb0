"""Hierarchical training with shared launches for the fine clusterings against the sequential form (taken when snapshots are
asked for): the same decisions; sums differ by their order only."""
import numpy as np
import pytest

from tests import datagen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k,opts", [(30_000, 96, 200, {}), (12_001, 33, 120, {}), (20_000, 64, 150, dict(angular=1)), (20_000, 128, 64, dict(early_termination=1, tol=0.02)),
                                        (20_000, 130, 64, dict(early_termination=1, tol=0.05, angular=1)), (2_000, 130, 1_900, {})])
def test_shared_launches_decide_like_the_sequential_form(n, d, k, opts):
    import superkmeans_b200 as skm

    x = datagen.gaussian_mixture(n, d, max(8, k // 3), 0.3, n)
    res = []
    for trace in (True, False):
        e = skm.Engine(k, d, skm.default_config(True, **dict(dict(early_termination=0, suppress_warnings=1), **opts)), hierarchical=True)
        e.set_trace(trace)
        c = e.train(x)
        res.append((c, e.assignments(), [(s.iteration, s.objective) for s in e.stats(2)]))
    (c0, a0, s0), (c1, a1, s1) = res
    assert [i for i, _ in s0] == [i for i, _ in s1]
    o0, o1 = np.array([o for _, o in s0]), np.array([o for _, o in s1])
    scale = max(float(o0.max()), 1e-12)
    first = np.array([i for i, _ in s0]) == 1
    assert np.abs(o0 - o1)[first].max() <= 1e-5 * scale   # distances near zero carry the rounding of the norms
    assert np.abs(o0 - o1).max() <= 2e-2 * scale
    assert (a0 == a1).mean() >= 0.98
    assert a1.max() < k and np.isfinite(c1).all()


def _two_levels(n, d, groups, each, spread, seed):
    """Unit rows in `groups` groups of `each` clusters whose distances from each other are `spread` times those of the groups."""
    rng = np.random.default_rng(seed)
    c = np.repeat(rng.standard_normal((groups, d), dtype=np.float32), each, 0) + np.float32(spread) * rng.standard_normal((groups * each, d), dtype=np.float32)
    x = c[rng.integers(0, groups * each, n)] + np.float32(spread / 2) * rng.standard_normal((n, d), dtype=np.float32)
    return x / np.linalg.norm(x, axis=1, keepdims=True)


@pytest.mark.parametrize("n,d,spread", [(20_000, 96, 0.1), (20_000, 96, 3e-2), (20_000, 96, 1e-3), (20_001, 33, 1e-3), (20_000, 260, 0.0)])
def test_clusters_close_to_each_other(n, d, spread):
    import superkmeans_b200 as skm

    x = _two_levels(n, d, 14, 14, spread, n)
    res = []
    for trace in (True, False):
        e = skm.Engine(196, d, skm.default_config(True, early_termination=0, suppress_warnings=1), hierarchical=True)
        e.set_trace(trace)
        c = e.train(x)
        res.append([(s.iteration, s.objective) for s in e.stats(2)])
        assert np.isfinite(c).all()
    s0, s1 = res
    assert [i for i, _ in s0] == [i for i, _ in s1]
    # distances of unit rows by norms and products: a few roundings of 2 (|x|^2 + |c|^2) each
    per_row = 4 * 2.0 ** -23
    first = np.array([o for i, o in s0 if i == 1]), np.array([o for i, o in s1 if i == 1])
    assert np.abs(first[0] - first[1]).sum() <= per_row * n + 1e-5 * first[0].sum()
    # rows between coincident centroids fall either way, and splits follow from the sizes: alike, not equal
    last = [sum(o for i, o in s if i == 5) for s in (s0, s1)]
    assert abs(last[0] - last[1]) <= 0.1 * last[0] + per_row * n, last


def test_clusters_close_to_each_other_take_no_cliff():
    import superkmeans_b200 as skm

    n, d, k = 200_000, 256, 1_600
    times = []
    for spread in (0.3, 1e-3):
        x = _two_levels(n, d, 40, 40, spread, 1)
        e = skm.Engine(k, d, skm.default_config(True, early_termination=0, suppress_warnings=1), hierarchical=True)
        e.train(x)
        e = skm.Engine(k, d, skm.default_config(True, early_termination=0, suppress_warnings=1), hierarchical=True)
        e.train(x)
        times.append(e.phase_times()["search/1st_blas"][0])
    # every pair in fp32 on the second, one fp16 product per pair on the first; a row at a time it was 7.1 times as long
    # here and 10 at 2.5M x 768
    assert times[1] <= 4 * times[0], times


@pytest.mark.parametrize("spread", [0.3, 1e-3], ids=["few listed", "many listed"])
@pytest.mark.parametrize("value", [np.nan, np.inf, 3e38])
def test_a_row_without_a_distance(value, spread):
    import superkmeans_b200 as skm

    n, d, k = 20_000, 96, 196
    x = _two_levels(n, d, 14, 14, spread, 2)
    x[777, 5] = value
    res = []
    for trace in (True, False):
        e = skm.Engine(k, d, skm.default_config(True, early_termination=0, suppress_warnings=1, seed=3), hierarchical=True)
        e.set_trace(trace)
        e.train(x)
        res.append(np.array([s.objective for s in e.stats(2) if s.iteration == 1]))
        assert e.assignments().max() < k
    # the row counts for nothing, or (a finite one whose squared norm is not) for an infinity, in either form
    finite = np.isfinite(res[0])
    np.testing.assert_array_equal(res[0][~finite], res[1][~finite])
    assert finite.sum() >= len(finite) - 1 and (finite.all() or value == 3e38)
    assert (np.abs(res[0] - res[1])[finite] <= 1e-5 * np.abs(res[0][finite]) + 1e-3).all(), res
