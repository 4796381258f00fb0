"""Host inputs and outputs, which cross in pinned pieces, against the same call on device arrays."""
import numpy as np
import pytest

from tests import datagen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k", [(1, 4, 1), (31, 3, 2), (70_001, 33, 40), (1_048_577, 4, 9), (43_700, 768, 30)])
def test_assign_from_host_equals_device(n, d, k):
    import torch

    import superkmeans_b200 as skm

    x = np.random.default_rng(n).standard_normal((n, d), dtype=np.float32)
    c = x[:k] + np.float32(0.01)
    e = skm.Engine(k, d)
    out = torch.empty(n, dtype=torch.int32, device="cuda")
    # (device arrays straight from the default stream: the call waits for it)
    e.assign(torch.from_numpy(x).cuda(), torch.from_numpy(c).cuda(), n=n, on_device=True, out=out)
    np.testing.assert_array_equal(e.assign(x, c).view(np.int32), out.cpu().numpy())


@pytest.mark.parametrize("hier", [False, True])
@pytest.mark.parametrize("fraction,rotated", [(0.5, 0), (0.5, 1), (1.0, 0), (1.0, 1)])
def test_train_from_host_equals_device(hier, fraction, rotated):
    import torch

    import superkmeans_b200 as skm

    n, d, k = 30_000, 96, 60
    x = datagen.gaussian_mixture(n, d, k, 0.3, 5)
    xd = torch.from_numpy(x).cuda()
    c = []
    for data, where in ((x, False), (xd, True)):
        cfg = skm.default_config(hier, sampling_fraction=fraction, max_points_per_cluster=10_000, data_already_rotated=rotated, early_termination=0, suppress_warnings=1)
        c.append(skm.Engine(k, d, cfg, hierarchical=hier).train(data, n=n, on_device=where))
    np.testing.assert_array_equal(c[0], c[1])


@pytest.mark.parametrize("n,d,k", [(300, 16, 20), (60_000, 64, 50), (20_000, 96, 2_000)])
def test_arrays_of_the_gpu_in_the_place_of_host_ones(n, d, k):
    import torch

    import superkmeans_b200 as skm
    from superkmeans_b200 import _lib

    x = np.random.default_rng(n).standard_normal((n, d), dtype=np.float32)
    c = x[:k].copy()
    e = skm.Engine(k, d)
    want = e.assign(x, c)
    xd, cd, out = torch.from_numpy(x).cuda(), torch.from_numpy(c).cuda(), torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    host = np.empty(n, dtype=np.uint32)
    _lib.check(_lib.lib.skm_assign(e._h, xd.data_ptr(), cd.data_ptr(), n, k, 0, host.ctypes.data), e._h)
    np.testing.assert_array_equal(host, want)
    _lib.check(_lib.lib.skm_assign(e._h, x.ctypes.data, c.ctypes.data, n, k, 0, out.data_ptr()), e._h)
    np.testing.assert_array_equal(out.cpu().numpy().view(np.uint32), want)
    model = []
    for data in (x.ctypes.data, xd.data_ptr()):
        model.append(np.empty((k, d), dtype=np.float32))
        e = skm.Engine(k, d, skm.default_config(False, sampling_fraction=0.5, max_points_per_cluster=100_000))
        _lib.check(_lib.lib.skm_train(e._h, data, n, 0, None, 0, model[-1]), e._h)
    np.testing.assert_array_equal(model[0], model[1])
