"""The plain kernel's selection against the oracle where it can go wrong: list
widths (k around 32, 64, 128 and 256), first tiles of fewer columns than k, ties at
the k-th distance across tiles and splits, distances that overflow or underflow
binary32, columns and rows past the last tile, unaligned and ragged dimensions."""
import numpy as np
import pytest

import holomap_b200 as hm
from parity import assert_same_bytes

pytestmark = pytest.mark.gpu
METRICS = ["euclidean", "cosine", "manhattan"]


def points(kind, n, d, seed=1):
    g = np.random.default_rng(seed)
    x = g.normal(size=(n, d))
    if kind == "ties":
        x = np.floor(g.uniform(0.0, 3.0, (n, d)))
    elif kind == "copies":  # more equal points than k: every list is cut inside a tie
        x = x[g.integers(0, 5, n)]
    elif kind == "huge":
        x[::3] *= 3e38 / np.abs(x[::3]).max()
    elif kind == "tiny":
        x *= 1e-30
        x[::4] *= 1e-13
    elif kind == "far":  # the nearest columns come last
        x *= np.linspace(9.0, 0.1, n)[:, None]
    return np.ascontiguousarray(x.astype(np.float32))


def check(oracle, x, k, metric, rows=None):
    n, d = x.shape
    knn = hm.exact_knn(x, d, k, metric, "plain")
    r0, r1 = rows or (0, n)
    oi, od = oracle.exact_knn(x, k, metric, rows=(r0, r1), threads=8)
    assert_same_bytes(knn.indices.reshape(n, k)[r0:r1], oi, "indices")
    assert_same_bytes(knn.dists.reshape(n, k)[r0:r1], od, "dists")


@pytest.mark.parametrize("metric", METRICS)
@pytest.mark.parametrize("k", [1, 31, 32, 33, 64, 65, 128, 129, 256])
def test_list_widths(oracle, metric, k):
    check(oracle, points("normal", 389, 19), k, metric)


@pytest.mark.parametrize("metric", METRICS)
@pytest.mark.parametrize("kind", ["ties", "copies", "huge", "tiny", "far"])
@pytest.mark.parametrize("n,d", [(257, 16), (1000, 33)])
def test_selection_edges(oracle, metric, kind, n, d):
    check(oracle, points(kind, n, d), 15, metric)


@pytest.mark.parametrize("n,d,k", [(1, 3, 1), (20, 4, 20), (128, 1, 30), (129, 17, 32), (6000, 20, 15), (6000, 20, 90)])
def test_shapes(oracle, n, d, k):
    check(oracle, points("normal", n, d), k, "euclidean", rows=(0, min(n, 200)) if n > 1000 else None)


@pytest.mark.parametrize("metric", METRICS)
@pytest.mark.parametrize("kind", ["near_one", "least", "zeros"])
@pytest.mark.parametrize("n", [353, 607])  # 31 and 1 places of the last row group without a row
def test_kth_distance_among_its_neighbours(oracle, metric, kind, n):
    """Distances one binary32 apart on both sides of the k-th, with ties, in no order of
    columns: around 1, among the least subnormals, and at 0 (more zero vectors than k,
    which under cosine are at distance 0 from every point)."""
    g = np.random.default_rng(n)
    x = np.zeros((n, 2), dtype=np.float32)
    if kind == "zeros":
        x[:] = g.normal(size=(n, 2))
        x[g.permutation(n)[: n // 3]] = 0.0
    else:
        # a few points at the origin (euclidean, manhattan) or on one axis (cosine), the
        # others a few steps of the last place around their k-th distance
        steps = g.integers(-4, 5, n)
        base = np.float32(1.0) if kind == "near_one" else np.float32(6e-45)
        x[:, 0] = (base.view(np.uint32).astype(np.int64) + steps).astype(np.uint32).view(np.float32)
        if metric == "cosine":
            x[:, 1] = 1.0 if kind == "near_one" else 1e-3
        x[g.permutation(n)[:5]] = (0.0, 1.0 if metric == "cosine" else 0.0)
    check(oracle, x, 15, metric)


def test_places_without_a_row_cost_nothing():
    """6,000 rows leave half of the last group's places empty, 6,016 none.  Letting
    every pair through there took the call from 390 to 910 us."""
    import torch
    from holomap_b200.device import DeviceKnnProblem
    best = {}
    for n in (6000, 6016):
        x = torch.rand(n, 24, generator=torch.Generator("cuda").manual_seed(1), device="cuda")
        p = DeviceKnnProblem(n, 24, 15, "cosine", "plain")
        times = []
        for _ in range(10):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            p.run(x)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        best[n] = min(times)
    assert best[6000] < 1.5 * best[6016]
