"""The dense chain on the tensor cores takes its points a slice at a time: memory for a last slice that is shorter than the others, and the
same answers however they are cut."""
import os
import subprocess

import numpy as np
import pytest

from tests import datagen

CPP = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpp")


def test_scratch_has_room_for_every_slice(tmp_path):
    exe = str(tmp_path / "slices_check")
    res = subprocess.run(["/usr/bin/g++", "-std=c++17", "-O1", "-Wall", os.path.join(CPP, "slices_check.cpp"), "-o", exe, "-lpthread"], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    res = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0 and "OK" in res.stdout, res.stdout + res.stderr


@pytest.fixture
def cut_at():
    from superkmeans_b200 import _lib, engine

    yield _lib.lib.skm_debug_chain_slice
    _lib.lib.skm_debug_chain_slice(0)
    engine.set_prune_split(0)


# 4864 points are 19 tiles, one more than share the SMs of a B200
@pytest.mark.gpu
@pytest.mark.parametrize("listed", [False, True], ids=["all points", "listed points"])
@pytest.mark.parametrize("rest", [0, 1, 255, 256, 4_608, 4_609])
def test_answers_do_not_depend_on_the_slices(cut_at, rest, listed):
    from superkmeans_b200 import engine

    d, k, n = 192, 1_300, 2 * 4_864 + rest
    x = datagen.gaussian_mixture(n, d, k // 4, 0.4, rest)
    y = datagen.gaussian_mixture(k, d, k // 4, 0.4, 7)
    prev = np.random.default_rng(rest).integers(0, k, n).astype(np.uint32)
    partial = engine.dimension_split(d)[1] // 2
    engine.set_prune_split(5 if listed else 3)   # 5: the lists overflow, their points are listed
    whole = engine.find_nearest_pruned(x, y, prev, partial)
    cut_at(4_864)
    cut = engine.find_nearest_pruned(x, y, prev, partial)
    cut_at(0)
    for a, b in zip(whole, cut):
        np.testing.assert_array_equal(a, b)
    engine.set_prune_split(2)
    want = engine.find_nearest_pruned(x, y, prev, partial)
    # pairs within rounding of a threshold of the search
    assert (cut[0] == want[0]).mean() >= 0.999
    exact = ((x.astype(np.float64) - y[cut[0]].astype(np.float64)) ** 2).sum(1)
    assert (np.abs(cut[1] - exact) <= 1e-5 * exact + 1e-12).all()
