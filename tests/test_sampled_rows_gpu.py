"""Rows that a Train samples from host memory, of whole cache lines and of parts of them, against the same rows on the device."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d", [(60_000, 16), (60_000, 32), (50_000, 33), (40_000, 156), (30_001, 57), (9_000, 1_040), (3, 5)])
def test_sampled_host_rows_are_the_rows_of_the_matrix(n, d):
    import torch

    import superkmeans_b200 as skm

    x = np.random.default_rng(d).standard_normal((n, d), dtype=np.float32)
    res = []
    for data, on_device in ((x, False), (torch.from_numpy(x).cuda(), True)):
        e = skm.Engine(2, d, skm.default_config(False, iters=2, sampling_fraction=0.7, early_termination=0, suppress_warnings=1))
        res.append((e.train(data, n=n, on_device=on_device), e.assignments()))
    assert (res[0][0] == res[1][0]).all() and (res[0][1] == res[1][1]).all()
