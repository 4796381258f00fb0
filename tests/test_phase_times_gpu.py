"""Phase times over many calls: all are counted, and none of the calls leaves its reading to a later one."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("where", ["host", "device"])
def test_many_short_calls(where):
    import torch

    import superkmeans_b200 as skm

    rng = np.random.default_rng(0)
    x, c = rng.standard_normal((64, 32), dtype=np.float32), rng.standard_normal((40, 32), dtype=np.float32)
    e = skm.Engine(40, 32)
    xd, cd, out = torch.from_numpy(x).cuda(), torch.from_numpy(c).cuda(), torch.empty(64, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    n = 3_500
    for _ in range(n):
        if where == "host":
            e.assign(x, c)
        else:
            e.assign(xd, cd, n=64, on_device=True, out=out)
    t = time.perf_counter()
    times = e.phase_times()
    t = time.perf_counter() - t
    assert times["search/1st_blas"][1] == n and times["search/1st_blas"][0] > 0
    assert t < 3e-3, t   # 3 us for each of the pairs that are left: 0.4 ms; 10 ms for all of them
