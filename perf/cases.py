"""Performance cases of the k-means engine: training, assignment and the allocation-free nearest-centroid call.

A case is a dict of plain values.  `listed()` gives the fixed ones, `draw()` further ones of the same ranges; `prepare()`
makes the inputs of a case on the GPU from a seed, `run()` makes one pass through the public entry points.

The rows stand in for unit-norm embeddings: a mixture in a low-dimensional latent space with a decaying spectrum and
unequal cluster sizes, mapped into d dimensions with a little noise in all of them.  Unlike isotropic noise in d
dimensions this leaves the clusters populated from iteration to iteration, as embeddings do.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import superkmeans_b200 as skm
from superkmeans_b200 import engine as eng

LATENT = 64          # dimensions the clusters live in
SPECTRUM = 0.6       # standard deviation of latent dimension j: (1 + j / 2) ** -SPECTRUM
WITHIN = 0.6         # spread inside a cluster against the spread of the centres
AMBIENT = 0.1        # norm of the noise over all d dimensions against the norm of a centre
CHUNK = 500_000      # rows made at a time


def listed():
    return [
        # ---- assignment: IVF lists looked up for queries, and whole collections added to an index
        # one query against the centroids, on the device: nothing but latency
        dict(name="assign_one_query", call="assign", n=1, k=1000, d=768, host=False),
        # a batch of queries in host memory, through the class a user of the Python package has
        dict(name="assign_query_batch", call="assign", n=1000, k=1000, d=768, host=True),
        # rows whose pitch is no multiple of 16 bytes, odd counts, host memory
        dict(name="assign_odd_host", call="assign", n=100_003, k=2_500, d=50, host=True),
        # a collection resident on the device added to a large index (benchmark configuration 5, fewer rows)
        dict(name="assign_collection", call="assign", n=2_000_000, k=16_384, d=384, host=False),
        # the call for programs that own all device memory; its sizes are those of its tests
        dict(name="nearest_in_pool", call="nearest", n=5_000, k=300, d=128, host=False),
        # assignment of the training rows to the trained centroids, started from the last iteration's answers
        dict(name="assign_training_points", call="training", n=300_000, k=1_000, d=768, host=False),
        # ---- training
        # the smallest useful problem: launches and set-up
        dict(name="train_tiny", call="train", n=2_000, k=20, d=64, host=True, hierarchical=False, sampling=0.0, angular=False, queries=0, early=True, iters=10),
        # the class with its defaults on 100 000 rows (flat, 30 % of the rows sampled, early stopping)
        dict(name="train_default", call="train", n=100_000, k=1_000, d=768, host=True, hierarchical=False, sampling=0.0, angular=False, queries=0, early=True, iters=10),
        # an odd width, unit centroids, recall followed with query vectors, all rows
        dict(name="train_odd_angular", call="train", n=30_001, k=300, d=130, host=True, hierarchical=False, sampling=1.0, angular=True, queries=200, early=True, iters=10),
        # benchmark configuration 2 (wide rows), fewer rows, device resident
        dict(name="train_wide", call="train", n=250_000, k=2_048, d=1_536, host=False, hierarchical=False, sampling=1.0, angular=False, queries=0, early=False, iters=10),
        # the headline configuration's width and iterations at a tenth of its rows, device resident
        dict(name="train_flat_large", call="train", n=1_000_000, k=4_000, d=1_024, host=False, hierarchical=False, sampling=1.0, angular=False, queries=0, early=False, iters=10),
        # the two-level algorithm (width and points per cluster of benchmark configuration 4), device resident
        dict(name="train_hierarchical", call="train", n=300_000, k=2_500, d=768, host=False, hierarchical=True, sampling=1.0, angular=False, queries=0, early=False, iters=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, lo, hi):
    """A row width: usually a multiple of 4 (rows that 16-byte loads can address), one in five as it falls."""
    d = _log_int(rng, lo, hi)
    return d if rng.random() < 0.2 else max(4, d // 4 * 4)


def draw(rng):
    call = rng.choice(["assign", "assign", "nearest", "training", "train", "train", "train", "hierarchical"])
    if call == "assign":
        host = rng.random() < 0.5
        d, k = _width(rng, 16, 1_536), _log_int(rng, 16, 16_384)
        most = min(2_000_000, (1.2e13 if d % 4 == 0 else 5e11) / (k * d), (1e8 if host else 1e9) / d)
        return dict(call="assign", n=_log_int(rng, 1, max(2, most)), k=k, d=d, host=host)
    if call == "nearest":
        d, k = _width(rng, 16, 1_024), _log_int(rng, 16, 8_192)
        return dict(call="nearest", n=_log_int(rng, 1, min(200_000, (2e12 if d % 4 == 0 else 2e11) / (k * d))), k=k, d=d, host=False)
    if call == "training":
        d, k = max(132, _width(rng, 132, 1_024)), _log_int(rng, 300, 2_000)
        n = _log_int(rng, 60 * k, max(61 * k, min(400_000, (5e11 if d % 4 == 0 else 5e10) / (k * d))))
        return dict(call="training", n=n, k=k, d=d, host=rng.random() < 0.5 and n * d <= 1e8)
    if call == "train":
        d, k = _width(rng, 32, 1_536), _log_int(rng, 8, 4_000)
        host = rng.random() < 0.5
        sampling = rng.choice([0.0, 1.0, 1.0])
        per = 200 if sampling == 0.0 else 60
        most = min(1_000_000, (4e12 if d % 4 == 0 else 1e11) / (k * d), (1e8 if host else 1e9) / d)
        k = min(k, max(8, int(most / (2 * per))))
        return dict(call="train", n=_log_int(rng, max(500, per * k), max(1_000, most)), k=k, d=d, host=host, hierarchical=False, sampling=sampling,
                    angular=rng.random() < 0.3, queries=rng.choice([0, 0, 100]) if host else 0, early=rng.random() < 0.5, iters=rng.choice([5, 10]))
    d, k = max(64, _width(rng, 64, 1_024)), _log_int(rng, 200, 2_500)
    n = _log_int(rng, 100 * k, max(101 * k, min(300_000, (8e12 if d % 4 == 0 else 5e11) / (k * d))))
    return dict(call="train", n=n, k=k, d=d, host=rng.random() < 0.3 and n * d <= 1e8, hierarchical=True, sampling=1.0, angular=rng.random() < 0.2, queries=0, early=False, iters=8)


class _Rows:
    """Unit rows around `k` centres, made on the GPU."""

    def __init__(self, k, d, seed):
        self.g = torch.Generator(device="cuda").manual_seed(seed)
        self.d = d
        m = min(d, LATENT)
        self.scale = (1.0 + torch.arange(m, device="cuda", dtype=torch.float32) / 2.0) ** -SPECTRUM
        self.norm = float(self.scale.norm())
        self.basis = torch.randn(m, d, generator=self.g, device="cuda") / math.sqrt(d)
        self.centres = torch.randn(k, m, generator=self.g, device="cuda") * self.scale
        # summed on the host in float64: the same labels from the same seed
        ends = torch.cumsum(torch.exp(0.7 * torch.randn(k, generator=self.g, device="cuda")).double().cpu(), 0)
        self.ends = (ends / ends[-1]).cuda()

    def __call__(self, n):
        x = torch.empty(n, self.d, device="cuda")
        for lo in range(0, n, CHUNK):
            part = x[lo:lo + CHUNK]
            at = torch.rand(part.shape[0], generator=self.g, device="cuda", dtype=torch.float64)
            labels = torch.searchsorted(self.ends, at, right=True).clamp_(max=self.ends.shape[0] - 1)
            latent = self.centres[labels] + WITHIN * self.scale * torch.randn(part.shape[0], self.scale.shape[0], generator=self.g, device="cuda")
            torch.matmul(latent, self.basis, out=part)
            part += (AMBIENT * self.norm / math.sqrt(self.d)) * torch.randn(part.shape, generator=self.g, device="cuda")
            part /= part.norm(dim=1, keepdim=True)
        return x

    def centroids(self):
        c = self.centres @ self.basis
        return c / c.norm(dim=1, keepdim=True)


def _host(t):
    return np.ascontiguousarray(t.cpu().numpy())


def _config(case):
    """The engine's configuration of a device-resident training case."""
    cfg = dict(angular=int(case["angular"]), early_termination=int(case["early"]))
    if case["sampling"]:
        cfg["sampling_fraction"] = case["sampling"]
    if not case["hierarchical"]:
        cfg["iters"] = case["iters"]
    return cfg


def prepare(case, seed):
    call, n, k, d = case["call"], case["n"], case["k"], case["d"]
    rows = _Rows(k, d, seed)
    state = dict(case, x=rows(n))
    if call == "assign":
        c = rows.centroids()
        if case["host"]:
            # the trained model such a program holds: the class needs one before it assigns
            model = skm.SuperKMeans(4, d, hierarchical=False, iters=1)
            model.train(_host(rows(64)))
            state.update(x=_host(state["x"]), c=_host(c), model=model)
        else:
            state.update(c=c, model=skm.Engine(k, d), out=torch.empty(n, dtype=torch.int32, device="cuda"))
    elif call == "nearest":
        state.update(c=rows.centroids(), knn=torch.empty(n, dtype=torch.int32, device="cuda"), dist=torch.empty(n, device="cuda"))
    elif call == "training":
        model = skm.Engine(k, d, skm.default_config(False, iters=3, sampling_fraction=1.0, early_termination=0))
        torch.cuda.synchronize()
        c = model.train(state["x"], n=n, on_device=True)
        if case["host"]:
            state.update(x=_host(state["x"]), c=c, model=model)
        else:
            state.update(c=torch.from_numpy(c).cuda(), model=model, out=torch.empty(n, dtype=torch.int32, device="cuda"))
    elif case["host"]:
        state["q"] = _host(rows(case["queries"])) if case["queries"] else None
        state["x"] = _host(state["x"])
    return state


def run(state):
    call, n, k, d, x = state["call"], state["n"], state["k"], state["d"], state["x"]
    if call == "nearest":
        eng.find_nearest_noalloc(x.data_ptr(), state["c"].data_ptr(), n, k, d, state["knn"].data_ptr(), state["dist"].data_ptr())
        return state["knn"], state["dist"]
    if call == "assign" or call == "training":
        fn = state["model"].assign if call == "assign" else state["model"].assign_training_points
        if state["host"]:
            return fn(x, state["c"])
        return fn(x, state["c"], n=n, on_device=True, out=state["out"])
    # a model trains once, so every pass makes its own
    if state["host"]:
        options = dict(sampling_fraction=state["sampling"]) if state["sampling"] else {}
        if not state["hierarchical"]:
            options["iters"] = state["iters"]
        model = skm.SuperKMeans(k, d, hierarchical=state["hierarchical"], angular=state["angular"], early_termination=state["early"], **options)
        c = model.train(x, queries=state["q"])
        stats = model.hierarchical_iteration_stats.fineclustering_iteration_stats if state["hierarchical"] else model.iteration_stats
        return dict(centroids=c, objective=float(stats[-1].objective))
    model = skm.Engine(k, d, skm.default_config(state["hierarchical"], **_config(state)), hierarchical=state["hierarchical"])
    c = model.train(x, n=n, on_device=True)
    return dict(centroids=c, assignments=model.assignments(), objective=float(model.stats(2 if state["hierarchical"] else 0)[-1].objective))


def work(case):
    call, n, k, d = case["call"], case["n"], case["k"], case["d"]
    rows = n
    if call == "train" and not case["sampling"]:
        rows = min(int(0.3 * n), 256 * k)
    nbytes = 4.0 * (rows * d + k * d)
    if call in ("assign", "nearest"):
        return {"bytes": nbytes + (4.0 if call == "assign" else 8.0) * n, "flops": 2.0 * n * k * d}
    # the search looks at the leading dimensions of every pair in all passes but the first
    leading = d if d < 128 or k <= 256 else eng.dimension_split(d)[1] / 2
    if call == "training":
        return {"bytes": nbytes + 4.0 * n, "flops": 2.0 * n * d * d + 2.0 * n * k * leading}
    rotations = 2.0 * (rows + 2 * k) * d * d
    if case["hierarchical"]:
        meso = math.sqrt(k)   # 3 passes over sqrt(k) coarse clusters, 5 over the sqrt(k) fine ones of each
        return {"bytes": nbytes + 4.0 * k * d, "flops": rotations + 8 * 2.0 * rows * meso * d}
    passes = 1 if case["early"] else case["iters"] - 1
    return {"bytes": nbytes + 4.0 * k * d, "flops": rotations + 2.0 * rows * k * (d + passes * leading)}


def tolerance(case):
    if case["call"] == "nearest":
        return {"rel": 1e-5, "max": 1e-4, "differ": 1e-4}      # fp32 distances; rows at the same distance from two centroids
    if case["call"] == "assign":
        return {"rel": 0.0, "differ": 1e-4}
    if case["call"] == "training":
        return {"rel": 0.0, "differ": 1e-3}    # pairs within rounding of a pruning threshold
    # Training repeats the assignment up to ten times: a row whose two nearest centroids tie to rounding moves two
    # centroids by 1 / (cluster size), which moves further rows.
    return {"rel": 1e-2, "max": 0.9, "differ": 1e-2}
