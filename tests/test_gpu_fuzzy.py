"""GPU parity of the fuzzy simplicial set (src/fuzzy.rs:25-91) against the
oracle's restatement, entry for entry and bit for bit, and against the
reference's own unit cases and golden fixtures."""
import ctypes
import json
from pathlib import Path

import numpy as np
import pytest

import holomap_b200 as hm
from holomap_b200._lib import check as check_rc
from parity import assert_same_bytes, edge_case

pytestmark = pytest.mark.gpu
GOLDEN = Path(__file__).resolve().parent / "golden"


def f32(x):
    return np.asarray(x, dtype=np.float32)


def check(oracle, idx, dist, sig, rho, k):
    g = hm.fuzzy_simplicial_set(hm.Knn(k, idx, dist), hm.SmoothKnn(sig, rho))
    rows, cols, vals = oracle.fuzzy_graph(idx, dist, sig, rho, k)
    assert g.n == idx.size // k
    assert_same_bytes(g.rows, rows, "rows")
    assert_same_bytes(g.cols, cols, "cols")
    assert_same_bytes(g.vals, vals, "vals")
    return g


def random_knn(n, k, seed):
    """A kNN-shaped graph: self first, then k - 1 distinct other points per
    row with ascending distances."""
    g = np.random.default_rng(seed)
    off = np.sort(g.integers(0, n - k + 1, size=(n, k - 1)), axis=1) + np.arange(k - 1) + 1
    idx = np.empty((n, k), dtype=np.uint32)
    idx[:, 0] = np.arange(n)
    idx[:, 1:] = (np.arange(n)[:, None] + off) % n
    dist = np.zeros((n, k), dtype=np.float32)
    dist[:, 1:] = np.sort(g.gamma(2.0, 1.0, size=(n, k - 1)).astype(np.float32), axis=1)
    return idx.reshape(-1), dist.reshape(-1)


def test_reference_line_points(oracle):
    # src/fuzzy.rs:97-129
    g = check(oracle, np.array([0, 1, 2, 1, 0, 2, 2, 1, 0], dtype=np.uint32),
              f32([0.0, 1.0, 3.0, 0.0, 1.0, 2.0, 0.0, 2.0, 3.0]),
              f32([3.72998046875, 1.864990234375, 1.864990234375]), f32([1.0, 1.0, 2.0]), 3)
    assert g.rows.tolist() == [0, 0, 1, 1, 2, 2]
    assert g.cols.tolist() == [1, 2, 0, 2, 0, 1]


def test_reference_one_directional_edge(oracle):
    # src/fuzzy.rs:131-155
    g = check(oracle, np.array([0, 1, 1, 2, 2, 1], dtype=np.uint32),
              f32([0.0, 1.0, 0.0, 0.1, 0.0, 0.1]), f32([1.0, 1.0, 1.0]), f32([0.5, 0.1, 0.1]), 2)
    w = oracle.expf(f32([-0.5]))[0]
    assert g.rows.tolist() == [0, 1, 1, 2]
    assert g.cols.tolist() == [1, 0, 2, 1]
    assert g.vals.tolist() == [w, w, 1.0, 1.0]


@pytest.mark.parametrize("name", ["blobs_euclidean", "cosine", "duplicates_euclidean"])
def test_golden_fixtures(oracle, name):
    # src/fixture_parity.rs:101-117 on the GPU's own kNN + smooth-kNN output
    fx = json.loads((GOLDEN / f"stage2_{name}.json").read_text())
    x = np.asarray(fx["data"], dtype=np.float32)
    k = fx["n_neighbors"]
    knn, sm = hm.knn_smooth(x, x.shape[1], k, fx["metric"])
    g = check(oracle, knn.indices, knn.dists, sm.sigmas, sm.rhos, k)
    assert g.rows.tolist() == fx["graph_rows"]
    assert g.cols.tolist() == fx["graph_cols"]
    e = np.asarray(fx["graph_vals"], dtype=np.float64)
    assert (np.abs(g.vals - e) <= 1e-5 * (1 + np.abs(e))).all()


@pytest.mark.parametrize("kind", ["gauss", "duplicates", "zeros", "huge", "grid", "sorted_line"])
@pytest.mark.parametrize("metric", ["euclidean", "cosine"])
def test_after_knn_edge_cases(oracle, kind, metric):
    # zero distances (d <= rho), sigma floors, zero vectors, tied neighbours
    x = edge_case(kind, 1500, 6, seed=5)
    knn, sm = hm.knn_smooth(x, 6, 15, metric)
    check(oracle, knn.indices, knn.dists, sm.sigmas, sm.rhos, 15)


@pytest.mark.parametrize("n,k", [(1, 1), (2, 2), (5, 5), (300, 1), (3000, 7), (65535, 4),
                                 (65536, 4), (200000, 15)])
def test_random_graphs(oracle, n, k):
    # the reverse copies are sorted on the bits of n: 16 up to n = 65535, 17
    # (a third radix pass) from n = 65536
    if k > n:
        pytest.skip("k above n")
    idx, dist = random_knn(n, k, seed=n + k) if k > 1 else (np.arange(n, dtype=np.uint32),
                                                            np.zeros(n, np.float32))
    sm = hm.smooth_knn(dist, k)
    g = check(oracle, idx, dist, sm.sigmas, sm.rhos, k)
    if k == 1:
        assert g.rows.size == 0  # only self edges
    key = g.rows.astype(np.uint64) << np.uint64(32) | g.cols
    assert (np.diff(key.astype(np.int64)) > 0).all()


def test_special_calibrations(oracle):
    # sigma == 0 rows, d <= rho, d - rho > 0 so large that expf underflows to
    # zero (dropped), +inf distances (weight 0, or 1 where sigma == 0), and
    # subnormal weights
    n, k = 4000, 8
    idx, dist = random_knn(n, k, seed=3)
    g = np.random.default_rng(4)
    sig = g.uniform(0.05, 2.0, size=n).astype(np.float32)
    rho = dist.reshape(n, k)[:, 1].copy()
    sig[::7] = 0.0
    rho[::11] = np.float32(1e30)
    d2 = dist.reshape(n, k)
    d2[::13, k // 2:] = np.float32(3e38)
    d2[5::17, 1:] = rho[5::17, None] + np.float32(95.0) * sig[5::17, None]
    d2[3::19, k - 1] = np.inf
    check(oracle, idx, dist, sig, rho, k)


def test_hub_rows(oracle):
    """Every row lists the same first points, so their reverse lists hold all
    n rows (in-degree n), next to rows of in-degree 0."""
    n, k = 5000, 6
    idx = np.empty((n, k), dtype=np.uint32)
    idx[:, 0] = np.arange(n)
    for r in range(n):
        others = [c for c in range(k + 1) if c != r][: k - 1]
        idx[r, 1:] = others
    dist = np.zeros((n, k), dtype=np.float32)
    dist[:, 1:] = np.linspace(0.5, 2.0, k - 1, dtype=np.float32)
    sm = hm.smooth_knn(dist.reshape(-1), k)
    g = check(oracle, idx.reshape(-1), dist.reshape(-1), sm.sigmas, sm.rhos, k)
    assert (g.rows == 0).sum() == n - 1


def test_device_entry_point_on_a_stream(oracle):
    """hm_fuzzy_graph_device on torch memory and a side stream equals the
    host entry point."""
    import ctypes
    import torch
    n, k = 20000, 12
    idx, dist = random_knn(n, k, seed=9)
    sm = hm.smooth_knn(dist, k)
    lib = hm.lib()
    ws_bytes = lib.hm_fuzzy_workspace_bytes(n, k)
    assert ws_bytes > 0
    dev = lambda a: torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda()
    d_idx, d_dist, d_sig, d_rho = dev(idx), dev(dist), dev(sm.sigmas), dev(sm.rhos)
    cap = 2 * n * k
    rows = torch.empty(cap, dtype=torch.int32, device="cuda")
    cols = torch.empty(cap, dtype=torch.int32, device="cuda")
    vals = torch.empty(cap, dtype=torch.float32, device="cuda")
    nnz = torch.zeros(1, dtype=torch.int64, device="cuda")
    ws = torch.empty(ws_bytes, dtype=torch.uint8, device="cuda")
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    for _ in range(2):
        check_rc(lib.hm_fuzzy_graph_device(d_idx.data_ptr(), d_dist.data_ptr(), d_sig.data_ptr(),
                                           d_rho.data_ptr(), n, k, rows.data_ptr(), cols.data_ptr(),
                                           vals.data_ptr(), nnz.data_ptr(), ws.data_ptr(), ws_bytes,
                                           ctypes.c_void_p(s.cuda_stream)))
    s.synchronize()
    m = int(nnz.item())
    r, c, v = oracle.fuzzy_graph(idx, dist, sm.sigmas, sm.rhos, k)
    assert m == r.size
    assert_same_bytes(rows[:m].cpu().numpy().view(np.uint32), r, "rows")
    assert_same_bytes(cols[:m].cpu().numpy().view(np.uint32), c, "cols")
    assert_same_bytes(vals[:m].cpu().numpy(), v, "vals")


def test_device_entry_point_reports_an_index_not_below_n(oracle):
    """hm_fuzzy_graph_device trusts no index: entries at or above n are
    dropped by the rows kernel (so every later access stays in bounds) and
    hm_fuzzy_graph_status reports them; the rest of the graph is the fuzzy
    set of the graph without those entries."""
    import ctypes
    import torch
    n, k = 3000, 10
    idx, dist = random_knn(n, k, seed=17)
    sm = hm.smooth_knn(dist, k)
    bad = idx.copy().reshape(n, k)
    bad[5, 3] = n          # just past the end
    bad[77, 9] = 0xFFFFFFF0  # far past it
    bad = bad.reshape(-1)
    lib = hm.lib()
    ws_bytes = lib.hm_fuzzy_workspace_bytes(n, k)
    dev = lambda a: torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda()
    d_idx, d_dist, d_sig, d_rho = dev(bad), dev(dist), dev(sm.sigmas), dev(sm.rhos)
    cap = 2 * n * k
    rows = torch.empty(cap, dtype=torch.int32, device="cuda")
    cols = torch.empty(cap, dtype=torch.int32, device="cuda")
    vals = torch.empty(cap, dtype=torch.float32, device="cuda")
    nnz = torch.zeros(1, dtype=torch.int64, device="cuda")
    ws = torch.empty(ws_bytes, dtype=torch.uint8, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    check_rc(lib.hm_fuzzy_graph_device(d_idx.data_ptr(), d_dist.data_ptr(), d_sig.data_ptr(),
                                       d_rho.data_ptr(), n, k, rows.data_ptr(), cols.data_ptr(),
                                       vals.data_ptr(), nnz.data_ptr(), ws.data_ptr(), ws_bytes,
                                       stream))
    assert lib.hm_fuzzy_graph_status(ws.data_ptr(), n, k, stream) == hm.HM_ERR_INVALID
    assert b"not below n" in lib.hm_last_error()
    m = int(nnz.item())
    assert 0 < m <= cap
    # the same graph with those two entries given strength 0 (dropped) and a
    # valid column, which the oracle drops the same way
    fixed_idx, fixed_dist = idx.copy(), dist.copy()
    r, c, v = oracle.fuzzy_graph(fixed_idx, fixed_dist, sm.sigmas, sm.rhos, k)
    got = set(zip(rows[:m].cpu().numpy().tolist(), cols[:m].cpu().numpy().tolist()))
    want = set(zip(r.tolist(), c.tolist()))
    assert got <= want  # only entries of the valid graph, none invented
    # a valid graph afterwards reports no error on the same workspace
    d_idx.copy_(dev(idx))
    check_rc(lib.hm_fuzzy_graph_device(d_idx.data_ptr(), d_dist.data_ptr(), d_sig.data_ptr(),
                                       d_rho.data_ptr(), n, k, rows.data_ptr(), cols.data_ptr(),
                                       vals.data_ptr(), nnz.data_ptr(), ws.data_ptr(), ws_bytes,
                                       stream))
    assert lib.hm_fuzzy_graph_status(ws.data_ptr(), n, k, stream) == hm.HM_OK
    assert int(nnz.item()) == r.size


def test_rows_at_the_sort_widths(oracle):
    """Hubs whose k + in-degree sits on and just past 64, 128, 256 and 512
    slots, the widths of the row kernels (the last one is the hub kernel's)."""
    n, k = 3000, 9
    indeg = [64 - k, 65 - k, 128 - k, 129 - k, 256 - k, 257 - k, 512 - k, 513 - k]
    idx = np.empty((n, k), dtype=np.uint32)
    for i in range(n):
        row = [i] + [j for j, m in enumerate(indeg) if 100 <= i < 100 + m and j != i]
        t = 1
        while len(row) < k:
            c = 100 + (i * 7 + t * 13) % (n - 100)
            if c not in row:
                row.append(c)
            t += 1
        idx[i] = row
    g = np.random.default_rng(3)
    dist = np.sort(g.gamma(2.0, 1.0, (n, k)).astype(np.float32), axis=1)
    dist[:, 0] = 0.0
    rho = dist[:, 1].copy()
    out = check(oracle, idx.reshape(-1), dist.reshape(-1), f32(np.full(n, 0.7)), rho, k)
    # node j < 8 lists no hub, so its row is its own k - 1 entries and its arrivals
    assert np.bincount(out.rows, minlength=n)[:8].max() >= 513 - k


@pytest.mark.parametrize("n,k,hubs", [
    (600000, 3, 2),          # hub rows of n entries, wider than one bitmap window
    ((1 << 23) + 3, 2, 0),   # column and slot no longer share a 32-bit sort key
])
def test_wide_columns(oracle, n, k, hubs):
    g = np.random.default_rng(n)
    i = np.arange(n)
    idx = np.empty((n, k), dtype=np.uint32)
    idx[:, 0] = i
    for j in range(1, k):
        # (the last columns by name, so that the widest keys occur)
        idx[:, j] = (n - j) if j <= hubs else (i + 1 + (j - 1) * (n // k) + g.integers(0, n // k - 1, n)) % n
    dist = np.sort(g.gamma(2.0, 1.0, (n, k)).astype(np.float32), axis=1)
    dist[:, 0] = 0.0
    for j in range(1, hubs + 1):  # a hub's own entry for itself would repeat its first
        idx[n - j, j] = j
    check(oracle, idx.reshape(-1), dist.reshape(-1), f32(np.ones(n)), dist[:, 1].copy(), k)


def ring(n, k):
    idx = ((np.arange(n, dtype=np.int64)[:, None] + np.arange(1, k + 1)) % n).astype(np.uint32)
    dist = np.tile(np.linspace(0.1, 1.0, k, dtype=np.float32), (n, 1))
    return idx.reshape(-1), dist.reshape(-1), np.full(n, 0.5, np.float32), np.full(n, 0.1, np.float32)


def test_host_calls_from_pooled_and_own_memory():
    """A call whose device memory is above the pooled size, between calls below it, and
    calls of several threads at once (each on its own stream): one ring of neighbours
    at several sizes, whose entries are known from a small one."""
    from concurrent.futures import ThreadPoolExecutor
    k = 15

    def run(n):
        idx, dist, sig, rho = ring(n, k)
        g = hm.fuzzy_simplicial_set(hm.Knn(k, idx, dist), hm.SmoothKnn(sig, rho))
        assert g.rows.size == 2 * n * k
        return g

    small = run(1000)
    middle = small.vals.reshape(1000, 2 * k)[500]  # columns in order: 15 before, 15 after
    for n in (260_000, 3000):
        g = run(n)
        assert np.array_equal(g.rows, np.repeat(np.arange(n, dtype=np.uint32), 2 * k))
        v = g.vals.reshape(n, 2 * k)[k:n - k]
        assert np.array_equal(v, np.broadcast_to(middle, v.shape))
    with ThreadPoolExecutor(4) as pool:
        for n, g in zip([2000, 5000, 2000, 9000] * 3, pool.map(run, [2000, 5000, 2000, 9000] * 3)):
            assert np.array_equal(g.vals.reshape(n, 2 * k)[k:n - k], np.broadcast_to(middle, (n - 2 * k, 2 * k)))
            pairs = hm.smallest_eigenpairs(g, 2)
            assert abs(float(pairs.values[0])) < 1e-9


class DeviceGraph:
    """hm_fuzzy_graph_device on torch memory: outputs with guard words behind
    them and a workspace full of ones (what an earlier call may have left)."""
    GUARD = 4096

    def __init__(self, n, k):
        import torch
        self.n, self.k, self.cap = n, k, 2 * n * k
        self.out = [torch.full((self.cap + self.GUARD,), -7, dtype=torch.int32, device="cuda") for _ in range(3)]
        self.nnz = torch.full((1,), -1, dtype=torch.int64, device="cuda")
        self.ws_bytes = hm.lib().hm_fuzzy_workspace_bytes(n, k)
        self.ws = torch.full((self.ws_bytes + self.GUARD,), 255, dtype=torch.uint8, device="cuda")

    def run(self, idx, dist, sig, rho):
        """Status of the graph; (nnz, rows, cols, vals) of the device arrays."""
        import torch
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).cuda()
        keep = [dev(a) for a in (idx, dist, sig, rho)]
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        check_rc(hm.lib().hm_fuzzy_graph_device(*[t.data_ptr() for t in keep], self.n, self.k,
                                                *[t.data_ptr() for t in self.out], self.nnz.data_ptr(),
                                                self.ws.data_ptr(), self.ws_bytes, stream))
        rc = hm.lib().hm_fuzzy_graph_status(self.ws.data_ptr(), self.n, self.k, stream)
        nnz = int(self.nnz.item())
        assert 0 <= nnz <= self.cap
        for t in self.out:
            assert bool((t[self.cap:] == -7).all()), "written past the outputs"
        assert bool((self.ws[self.ws_bytes:] == 255).all()), "written past the workspace"
        return rc, [nnz] + [t[:nnz].cpu().numpy() for t in self.out]


@pytest.mark.parametrize("n", [100, 113, 114, 1000])  # n + k up to 128: no row of a valid graph is long
@pytest.mark.parametrize("repeaters", [3, 20, 99])     # slots of the repeated column: k + 15 each
def test_repeated_indices_are_refused_in_bounds(oracle, n, repeaters):
    """Rows that list one column k times over: its k + in-degree reaches the
    widths of all three row kernels (75, 315 and 1,500 slots), also where n + k
    would rule long rows out.  Both entry points answer HM_ERR_INVALID and write
    nothing outside their arrays; a valid graph on the same workspace follows."""
    k = 15
    idx, dist = random_knn(n, k, seed=n)
    sig, rho = f32(np.full(n, 0.7)), dist.reshape(n, k)[:, 1].copy()
    bad = idx.copy().reshape(n, k)
    bad[1:1 + repeaters] = 0
    g = DeviceGraph(n, k)
    rc, _ = g.run(bad.reshape(-1), dist, sig, rho)
    assert rc == hm.HM_ERR_INVALID and b"repeats" in hm.lib().hm_last_error()
    with pytest.raises(Exception, match="repeats"):
        hm.fuzzy_simplicial_set(hm.Knn(k, bad.reshape(-1), dist), hm.SmoothKnn(sig, rho))
    rc, (nnz, rows, cols, vals) = g.run(idx, dist, sig, rho)
    r, c, v = oracle.fuzzy_graph(idx, dist, sig, rho, k)
    assert rc == hm.HM_OK and nnz == r.size
    assert_same_bytes(rows.view(np.uint32), r, "rows")
    assert_same_bytes(cols.view(np.uint32), c, "cols")
    assert_same_bytes(vals.view(np.float32), v, "vals")


@pytest.mark.parametrize("n,k", [(1500, 3), (3000, 15), (2000, 100), (1300, 1100)])
def test_rows_that_list_the_same_points(oracle, n, k):
    """Every row lists the same k - 1 other points at the same places, which the
    entries' blocks count jointly: 1,024 entries are 342 rows, 69, 11 and part of one."""
    idx = np.empty((n, k), dtype=np.uint32)
    idx[:, 0] = np.arange(n)
    idx[:, 1:] = np.arange(k - 1)
    for r in range(k - 1):
        idx[r, 1:] = [c for c in range(k) if c != r]
    g = np.random.default_rng(k)
    dist = np.sort(g.gamma(2.0, 1.0, (n, k)).astype(np.float32), axis=1)
    dist[:, 0] = 0.0
    dist[::3, k - 1] = np.float32(3e38)  # strength 0
    check(oracle, idx.reshape(-1), dist.reshape(-1), f32(np.full(n, 0.7)), dist[:, 1].copy(), k)


@pytest.mark.parametrize("hubs", [1, 40, 74, 75, 160])
def test_hubs_shared_by_blocks(oracle, hubs):
    """Points that 600 rows or more list, over more columns than one window: one hub
    over all blocks, two blocks a hub with several windows each, and a block a hub (up
    to 74 and from 75 on with 148 blocks); more hubs than blocks.  A hub's own
    neighbours lie in every window, some listing it back, some with strength 0."""
    n, k, per = 140_003, 13, 600
    g = np.random.default_rng(hubs)
    hub = (37 + np.arange(hubs) * (n // hubs)).astype(np.int64)
    idx = (np.arange(n)[:, None] + np.arange(k)) % n  # itself and the next points
    lists = [[] for _ in range(n)]
    rows = g.permutation(n)
    for h in range(hubs):
        for r in rows[(h * per // 4 + np.arange(per)) % n]:  # about four hubs a row
            lists[r].append(hub[h])
    for h in hub:  # neighbours over the whole range, half of them listing the hub
        away = g.choice(n, k - 1, replace=False)
        lists[h] = [a for a in away if a != h]
        for a in away[::2]:
            lists[a].append(h)
    for r, extra in enumerate(lists):
        if extra:
            extra = [c for c in dict.fromkeys(extra) if c != r][: k - 1]
            rest = [c for c in idx[r, 1:] if c not in extra]
            idx[r] = [r] + (extra + rest)[: k - 1]
    dist = np.sort(g.gamma(2.0, 1.0, (n, k)).astype(np.float32), axis=1)
    dist[:, 0] = 0.0
    dist[::5, k // 2:] = np.float32(3e38)
    dist[::5] = np.sort(dist[::5], axis=1)
    out = check(oracle, idx.astype(np.uint32).reshape(-1), dist.reshape(-1), f32(np.full(n, 0.7)), dist[:, 1].copy(), k)
    assert (np.bincount(out.rows, minlength=n)[hub] > 512 - k).all()
