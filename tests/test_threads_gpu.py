"""Two threads with engines of their own on one GPU: they share parked memory, streams and events, and nothing else."""
import threading

import numpy as np
import pytest

from tests import datagen

pytestmark = pytest.mark.gpu


def test_two_threads():
    import superkmeans_b200 as skm

    jobs = [(6_000, 64, 50, False), (30_000, 256, 400, False), (20_000, 96, 200, True), (9_000, 130, 300, False)]
    data = [datagen.gaussian_mixture(n, d, k // 2, 0.3, n) for n, d, k, _ in jobs]

    def run(i):
        n, d, k, hierarchical = jobs[i]
        e = skm.Engine(k, d, skm.default_config(hierarchical, early_termination=0, suppress_warnings=1), hierarchical=hierarchical)
        c = e.train(data[i])
        return c, e.assign(data[i], c)

    want = [run(i) for i in range(len(jobs))]
    wrong = []

    def worker(order):
        try:
            for i in order:
                c, a = run(i)
                if not (np.array_equal(c, want[i][0]) and np.array_equal(a, want[i][1])):
                    wrong.append(i)
        except Exception as e:   # (a thread's exception ends nobody but the thread)
            wrong.append(e)

    threads = [threading.Thread(target=worker, args=(order,)) for order in ([0, 1, 2, 3] * 4, [3, 2, 1, 0, 1] * 3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong
