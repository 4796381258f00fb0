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
