"""GPU parity of the screened paths (tcgen05 BF16 / TF32 / split-BF16 screen +
exact rerank): every path must return the oracle's bytes; the screen itself
must stay inside its proven band."""
import numpy as np
import pytest

import holomap_b200 as hm
from parity import assert_same_bytes, edge_case, rows_sorted_by_key

pytestmark = pytest.mark.gpu
PATHS = ["screen_bf16", "screen_tf32", "screen_bf16x3"]


def screened_values(x, metric, path):
    """Run one screened call with the dump hook set; return c^ (n x n)."""
    import torch
    n, d = x.shape
    buf = torch.full((n * n,), float("nan"), dtype=torch.float32, device="cuda")
    hm.lib().hm_debug_set_screen_dump(buf.data_ptr())
    try:
        hm.exact_knn(x, d, 5, metric, path)
    finally:
        hm.lib().hm_debug_set_screen_dump(None)
    return buf.cpu().numpy().reshape(n, n)


@pytest.mark.parametrize("path", PATHS)
@pytest.mark.parametrize("metric", ["cosine", "euclidean"])
def test_screen_values_track_exact_inner_products(path, metric):
    g = np.random.default_rng(1)
    n, d = 700, 72
    x = g.normal(size=(n, d)).astype(np.float32)
    c = screened_values(x, metric, path)
    xd = x.astype(np.float64)
    if metric == "cosine":
        u = xd / np.linalg.norm(xd, axis=1, keepdims=True)
        exact = 1.0 - u @ u.T
        tol = {"screen_bf16": 2e-2, "screen_tf32": 3e-3, "screen_bf16x3": 1e-4}[path]
    else:
        u = xd - xd.mean(0)
        m = np.sqrt((u * u).sum(1).max())
        u = u * 2.0 ** -np.frexp(m)[1]
        sq = (u * u).sum(1)
        exact = sq[:, None] + sq[None, :] - 2 * u @ u.T
        tol = {"screen_bf16": 2e-2, "screen_tf32": 3e-3, "screen_bf16x3": 1e-4}[path] * 4
    np.fill_diagonal(exact, 0.0)
    assert np.isfinite(c).all(), "screen left entries unwritten"
    err = np.abs(c - exact).max()
    assert err < tol, f"max |c^ - c| = {err}"


@pytest.mark.parametrize("path", PATHS)
@pytest.mark.parametrize("metric", ["euclidean", "cosine"])
@pytest.mark.parametrize("n,d,k", [(300, 5, 15), (1000, 50, 15), (4500, 130, 30), (2100, 384, 64),
                                   (5000, 16, 2), (1300, 7, 33)])
def test_screened_matches_oracle(oracle, path, metric, n, d, k):
    x = edge_case("gauss", n, d, seed=n + d)
    st = hm.HmStats()
    knn, sm = hm.knn_smooth(x, d, k, metric, path, stats=st)
    oi, od = oracle.exact_knn(x, k, metric)
    assert_same_bytes(knn.indices, oi, "indices")
    assert_same_bytes(knn.dists, od, "dists")
    osig, orho = oracle.smooth_knn(od, k)
    assert_same_bytes(sm.sigmas, osig, "sigma")
    assert_same_bytes(sm.rhos, orho, "rho")
    assert st.path_used == hm.KnnPath.parse(path)
    # every row is either reranked from at least k candidates or sent whole to
    # the exact fallback
    assert st.candidates_total >= (n - st.overflow_rows) * k


@pytest.mark.parametrize("path", PATHS)
@pytest.mark.parametrize("kind", ["duplicates", "ulp", "zeros", "huge", "tiny", "grid",
                                  "sorted_line"])
@pytest.mark.parametrize("metric", ["euclidean", "cosine"])
def test_screened_edge_cases(oracle, path, kind, metric):
    x = edge_case(kind, 1111, 6, seed=13)
    knn = hm.exact_knn(x, 6, 15, metric, path)
    oi, od = oracle.exact_knn(x, 15, metric)
    assert_same_bytes(knn.indices, oi, "indices")
    assert_same_bytes(knn.dists, od, "dists")


@pytest.mark.parametrize("name", ["blobs_euclidean", "cosine", "duplicates_euclidean"])
@pytest.mark.parametrize("path", PATHS)
def test_screened_golden_fixtures(oracle, name, path):
    import json
    from pathlib import Path
    fx = json.loads((Path(__file__).parent / "golden" / f"stage2_{name}.json").read_text())
    x = np.asarray(fx["data"], dtype=np.float32)
    k = fx["n_neighbors"]
    knn = hm.exact_knn(x, x.shape[1], k, fx["metric"], path)
    assert knn.indices.reshape(-1, k).tolist() == fx["knn_indices"]
    oi, od = oracle.exact_knn(x, k, fx["metric"])
    assert_same_bytes(knn.dists, od, "dists")


def test_screened_equals_plain_on_clustered_duplicates():
    from holomap_b200.synth import dups_20k
    wl = dups_20k(n=12000, d=64)
    a = hm.exact_knn(wl.data, wl.d, wl.k, wl.metric, "plain")
    for path in PATHS:
        st = hm.HmStats()
        b = hm.exact_knn(wl.data, wl.d, wl.k, wl.metric, path, stats=st)
        assert_same_bytes(b.indices, a.indices, f"{path} indices")
        assert_same_bytes(b.dists, a.dists, f"{path} dists")
        assert rows_sorted_by_key(b.indices.reshape(-1, wl.k), b.dists.reshape(-1, wl.k))


@pytest.mark.parametrize("path", PATHS)
def test_device_data_at_a_4_byte_offset(oracle, path):
    """The C ABI takes any 4-byte-aligned device pointer: points given at an
    odd float offset inside a larger buffer (d a multiple of 4, so the
    rerank's 16-byte row loads must not be used) return the oracle's bytes."""
    import torch
    from holomap_b200.device import DeviceKnnProblem
    n, d, k = 1500, 32, 15
    x = edge_case("gauss", n, d, seed=41)
    big = torch.zeros(n * d + 1, dtype=torch.float32, device="cuda")
    big[1:] = torch.from_numpy(x.reshape(-1)).cuda()
    view = big[1:].view(n, d)
    assert view.data_ptr() % 16 != 0
    p = DeviceKnnProblem(n, d, k, "euclidean", path)
    p.run(view)
    torch.cuda.synchronize()
    oi, od = oracle.exact_knn(x, k, "euclidean")
    assert_same_bytes(p.idx.cpu().numpy().view(np.uint32), oi, "indices")
    assert_same_bytes(p.dist.cpu().numpy(), od, "dists")
    assert p.stats().path_used == hm.KnnPath.parse(path)


@pytest.mark.parametrize("path", PATHS)
@pytest.mark.parametrize("metric", ["euclidean", "cosine"])
@pytest.mark.parametrize("n", [2600, 3000])
def test_full_and_symmetric_emission_agree_with_the_oracle(oracle, path, metric, n):
    """The emission pass over every column tile (hm_tuning_symmetric(0)) and
    over the tiles on and above the diagonal only (hm_tuning_symmetric(1),
    whose rows also take candidates as columns), each with one CTA per
    128-row block and in the 2-SM form, return the oracle's bytes; the zero
    rows under cosine exercise the column side's general (non raw-product)
    test, and n = 3000 ends inside a 256-row block's second half."""
    lib = hm.lib()
    x = edge_case("zeros" if metric == "cosine" else "duplicates", n, 40, seed=5)
    x[::7] += 0.5  # keep most rows non-zero
    oi, od = oracle.exact_knn(x, 15, metric)
    osig, orho = oracle.smooth_knn(od, 15)
    for sym in (0, 1):
        for pair in (0, 1):
            assert lib.hm_tuning_symmetric(sym) == 0
            assert lib.hm_tuning_pair(pair) == 0
            try:
                st = hm.HmStats()
                knn, sm = hm.knn_smooth(x, 40, 15, metric, path, stats=st)
            finally:
                lib.hm_tuning_symmetric(-1)
                lib.hm_tuning_pair(-1)
            what = f"sym={sym} pair={pair}"
            assert_same_bytes(knn.indices, oi, f"{what} indices")
            assert_same_bytes(knn.dists, od, f"{what} dists")
            assert_same_bytes(sm.sigmas, osig, f"{what} sigma")
            assert_same_bytes(sm.rhos, orho, f"{what} rho")


@pytest.mark.parametrize("path", PATHS)
@pytest.mark.parametrize("n", [200, 1000, 2600])
def test_pair_and_single_cta_emission_agree_with_the_oracle(oracle, path, n):
    """The emission pass in the 2-SM form (hm_tuning_pair(1): a cluster of two
    CTAs shares one 256-row MMA, each loading half of every column tile) and
    with one CTA per 128-row block (hm_tuning_pair(0)) return the oracle's bytes,
    including a last 256-row block that ends inside its first half (n = 200,
    1000) and one whose second half lies past every row (n = 2600)."""
    lib = hm.lib()
    x = edge_case("duplicates", n, 40, seed=n)
    oi, od = oracle.exact_knn(x, 15, "euclidean")
    osig, orho = oracle.smooth_knn(od, 15)
    for pair in (0, 1):
        assert lib.hm_tuning_pair(pair) == 0
        try:
            knn, sm = hm.knn_smooth(x, 40, 15, "euclidean", path)
        finally:
            lib.hm_tuning_pair(-1)
        assert_same_bytes(knn.indices, oi, f"pair={pair} indices")
        assert_same_bytes(knn.dists, od, f"pair={pair} dists")
        assert_same_bytes(sm.sigmas, osig, f"pair={pair} sigma")
        assert_same_bytes(sm.rhos, orho, f"pair={pair} rho")


def _tight_clusters(n, d, seed, sigma=0.05):
    """Eight clusters far tighter than a BF16 or TF32 operand's rounding
    relative to their distance from the origin (the coarse screens' hard case)."""
    g = np.random.default_rng(seed)
    centres = g.normal(0.0, 4.0, size=(8, d))
    labels = g.integers(0, 8, size=n)
    return np.ascontiguousarray((centres[labels] + g.normal(0.0, sigma, size=(n, d))).astype(np.float32))


@pytest.mark.parametrize("metric", ["cosine", "euclidean"])
def test_auto_escalates_on_clusters_tighter_than_the_screen(metric):
    """A job left to the autotuner, whose choice here is the BF16 (cosine) or
    TF32 (euclidean) screen, hands over to its split-BF16 copy when the
    coarse screen's band swamps the rows' thresholds; the bytes equal the
    plain path's either way (escalation off: the coarse screen's own, slow
    but exact, result)."""
    lib = hm.lib()
    n, d, k = 4096, 384, 15
    x = _tight_clusters(n, d, seed=7)
    assert hm.autotune_path(n, d, k, metric) in (hm.KnnPath.SCREEN_BF16, hm.KnnPath.SCREEN_TF32)
    plain, psm = hm.knn_smooth(x, d, k, metric, "plain")
    st = hm.HmStats()
    knn, sm = hm.knn_smooth(x, d, k, metric, "auto", stats=st)
    assert st.path_used == int(hm.KnnPath.SCREEN_BF16X3), st.path_used
    for a, b, what in ((knn.indices, plain.indices, "indices"), (knn.dists, plain.dists, "dists"),
                       (sm.sigmas, psm.sigmas, "sigma"), (sm.rhos, psm.rhos, "rho")):
        assert_same_bytes(a, b, f"escalated {what}")
    assert lib.hm_tuning_escalation(0) == 0
    try:
        st0 = hm.HmStats()
        knn0, sm0 = hm.knn_smooth(x, d, k, metric, "auto", stats=st0)
    finally:
        lib.hm_tuning_escalation(1)
    assert st0.path_used == int(hm.autotune_path(n, d, k, metric))
    assert_same_bytes(knn0.indices, plain.indices, "coarse indices")
    assert_same_bytes(knn0.dists, plain.dists, "coarse dists")


def test_auto_keeps_the_coarse_screen_on_embedding_shaped_data():
    """Embedding-shaped data (the autotuner's cosine family) keeps the BF16
    screen: its band is a few percent of the rows' thresholds."""
    from holomap_b200.synth import embed_50k
    wl = embed_50k(n=8192)
    assert hm.autotune_path(wl.n, wl.d, wl.k, wl.metric) == hm.KnnPath.SCREEN_BF16
    plain, _ = hm.knn_smooth(wl.data, wl.d, wl.k, wl.metric, "plain")
    st = hm.HmStats()
    knn, _ = hm.knn_smooth(wl.data, wl.d, wl.k, wl.metric, "auto", stats=st)
    assert st.path_used == int(hm.KnnPath.SCREEN_BF16)
    assert_same_bytes(knn.indices, plain.indices, "indices")
    assert_same_bytes(knn.dists, plain.dists, "dists")


def test_batch_escalates_only_the_job_that_needs_it():
    """In one batch, the tightly clustered job escalates and the
    embedding-shaped one does not; both return the plain path's bytes."""
    import torch
    from holomap_b200.device import DeviceBatch
    from holomap_b200.synth import embed_50k
    a = _tight_clusters(4096, 384, seed=3)
    b = embed_50k(n=4096).data
    batch = DeviceBatch([(torch.from_numpy(a).cuda(), 15, "cosine"), (torch.from_numpy(b).cuda(), 30, "cosine")])
    batch.run()
    torch.cuda.synchronize()
    for j, (x, k) in enumerate(((a, 15), (b, 30))):
        plain, psm = hm.knn_smooth(x, 384, k, "cosine", "plain")
        idx, dist, sig, rho = batch.result(j)
        assert_same_bytes(idx.reshape(-1), plain.indices, f"job {j} indices")
        assert_same_bytes(dist.reshape(-1), plain.dists, f"job {j} dists")
        assert_same_bytes(sig, psm.sigmas, f"job {j} sigma")
        assert_same_bytes(rho, psm.rhos, f"job {j} rho")
    paths = [batch.stats(j).path_used for j in range(2)]
    assert paths[0] == int(hm.KnnPath.SCREEN_BF16X3), paths
    assert paths[1] != int(hm.KnnPath.SCREEN_BF16X3), paths


@pytest.mark.parametrize("n", [7999, 8001])
@pytest.mark.parametrize("metric", ["euclidean", "cosine"])
@pytest.mark.parametrize("d", [37, 64])
def test_rerank_of_mixed_magnitudes(oracle, n, metric, d):
    """The exact rerank on both sides of its change of rows per warp (8,000
    rows), on rows that mix signed zeros, subnormals, tiny and large values in
    odd and even dimensions (the cosine's odd dimensions take another exact
    conversion)."""
    g = np.random.default_rng(n + d)
    x = g.normal(size=(n, d)).astype(np.float32)
    x[::3, ::5] = -0.0
    x[1::3, 1::4] = np.float32(1e-40) * g.integers(-9, 9, x[1::3, 1::4].shape).astype(np.float32)
    x[2::5, 3::7] *= np.float32(1e-30)
    x[::7, 2::9] *= np.float32(64.0)
    k = 12
    knn = hm.exact_knn(x, d, k, metric, "screen_bf16x3")
    for r0 in (0, 4000, n - 96):
        oi, od = oracle.exact_knn(x, k, metric, rows=(r0, r0 + 96), threads=8)
        assert_same_bytes(knn.indices.reshape(n, k)[r0:r0 + 96], oi, f"indices {r0}")
        assert_same_bytes(knn.dists.reshape(n, k)[r0:r0 + 96], od, f"dists {r0}")


@pytest.mark.parametrize("sizes", [(5003,), (9000, 4100, 6000)])
def test_auto_escalates_where_the_band_spans_the_nearest_neighbours(sizes):
    """Gaussian mixtures under cosine at d = 300: the BF16 band is well below
    half of the thresholds but spans most of a row's nearest neighbours, so the
    split-BF16 copies take over, alone and in a batch (whose copies lie in their
    originals' candidate room); the bytes are the plain path's, no row overflows."""
    import torch
    from holomap_b200.device import DeviceBatch
    from holomap_b200.synth import gaussian_mixture
    d, k = 300, 15
    g = np.random.default_rng(11)
    data = [gaussian_mixture(g, n, d, 12, 4.0, 0.3, 3.0).astype(np.float32) for n in sizes]
    batch = DeviceBatch([(torch.from_numpy(x).cuda(), k, "cosine") for x in data])
    batch.run()
    torch.cuda.synchronize()
    for j, x in enumerate(data):
        plain, psm = hm.knn_smooth(x, d, k, "cosine", "plain")
        idx, dist, sig, rho = batch.result(j)
        assert_same_bytes(idx.reshape(-1), plain.indices, f"job {j} indices")
        assert_same_bytes(dist.reshape(-1), plain.dists, f"job {j} dists")
        assert_same_bytes(sig, psm.sigmas, f"job {j} sigma")
        assert_same_bytes(rho, psm.rhos, f"job {j} rho")
        st = batch.stats(j)
        if hm.autotune_path(x.shape[0], d, k, "cosine", batched=len(sizes) > 1) == hm.KnnPath.SCREEN_BF16:
            assert st.path_used == int(hm.KnnPath.SCREEN_BF16X3)
        assert st.overflow_rows == 0


@pytest.mark.parametrize("n", [150, 1500, 5000])
@pytest.mark.parametrize("path", ["screen_bf16", "screen_bf16x3"])
def test_selection_at_the_edges_of_its_register_widths(path, n):
    """k around the select's sort widths (32 and 64 keys; 64 is the screened paths'
    limit); a row's candidates number from k up to all of the rows."""
    g = np.random.default_rng(n)
    x = g.normal(size=(n, 20)).astype(np.float32)
    x[n // 2:n // 2 + 40] = x[0]  # ties at distance zero
    for k in (1, 2, 31, 32, 33, 63, 64):
        plain = hm.exact_knn(x, 20, k, "euclidean", "plain")
        knn = hm.exact_knn(x, 20, k, "euclidean", path)
        assert_same_bytes(knn.indices, plain.indices, f"k {k} indices")
        assert_same_bytes(knn.dists, plain.dists, f"k {k} dists")


def test_batch_merges_only_its_split_jobs():
    """Exact jobs with and without column splits between screened jobs of both
    short and long rows: every job's bytes are those of the job alone."""
    import torch
    from holomap_b200.device import DeviceBatch
    g = np.random.default_rng(5)
    shapes = [(90, 8, 5, "manhattan"), (3000, 12, 15, "euclidean"), (700, 40, 20, "manhattan"),
              (33, 3, 4, "euclidean"), (2500, 100, 10, "cosine"), (1025, 70, 15, "euclidean"),
              (2000, 5, 7, "manhattan")]
    data = [g.normal(size=(n, d)).astype(np.float32) for n, d, _, _ in shapes]
    batch = DeviceBatch([(torch.from_numpy(x).cuda(), k, m) for x, (_, _, k, m) in zip(data, shapes)])
    batch.run()
    torch.cuda.synchronize()
    for j, (x, (n, d, k, m)) in enumerate(zip(data, shapes)):
        plain, psm = hm.knn_smooth(x, d, k, m, "plain")
        idx, dist, sig, rho = batch.result(j)
        assert_same_bytes(idx.reshape(-1), plain.indices, f"job {j} indices")
        assert_same_bytes(dist.reshape(-1), plain.dists, f"job {j} dists")
        assert_same_bytes(sig, psm.sigmas, f"job {j} sigma")
        assert_same_bytes(rho, psm.rhos, f"job {j} rho")


@pytest.mark.parametrize("path", PATHS)
@pytest.mark.parametrize("metric", ["euclidean", "cosine"])
@pytest.mark.parametrize("d", [1, 3, 8, 9, 16, 17, 32, 33, 63, 64, 65, 88, 127, 128, 129])
def test_operand_rows_of_every_length_class(path, metric, d):
    """Row lengths around the operand kernels' lanes per row (16, 32, 64), their
    4-element pieces, the split segments' 8 and the K steps of 16 and 8; the bytes
    are the plain path's and no row falls back for want of a bound."""
    g = np.random.default_rng(d)
    n, k = 333, 7
    x = (g.normal(size=(n, d)) + 3.0).astype(np.float32)
    plain = hm.exact_knn(x, d, k, metric, "plain")
    knn = hm.exact_knn(x, d, k, metric, path)
    assert_same_bytes(knn.indices, plain.indices, "indices")
    assert_same_bytes(knn.dists, plain.dists, "dists")


@pytest.mark.parametrize("seed_div", [1, 3, 8])
@pytest.mark.parametrize("metric", ["euclidean", "cosine"])
def test_threshold_chunks_of_every_width(seed_div, metric):
    """Sizes and k for which a row's chunk minima cover 4 columns up to 64 of several
    tiles, with a last part and a last chunk that are not full; fewer minima than k."""
    from holomap_b200 import _lib
    g = np.random.default_rng(seed_div)
    lib = _lib.lib()
    assert lib.hm_tuning_override(seed_div) == 0
    try:
        for n, k in ((40, 20), (130, 3), (257, 5), (700, 64), (1500, 21), (2049, 15), (4100, 41), (9001, 5), (20011, 12)):
            x = g.normal(size=(n, 10)).astype(np.float32)
            x[n // 3] = x[n // 2]
            plain = hm.exact_knn(x, 10, k, metric, "plain")
            knn = hm.exact_knn(x, 10, k, metric, "screen_bf16x3")
            assert_same_bytes(knn.indices, plain.indices, f"{n} {k} indices")
            assert_same_bytes(knn.dists, plain.dists, f"{n} {k} dists")
    finally:
        lib.hm_tuning_override(0)


@pytest.mark.parametrize("path", ["screen_bf16", "screen_bf16x3"])
@pytest.mark.parametrize("d", [10, 200])
def test_emission_ranges_of_one_job(path, d):
    """One job's emission units from one tile to several row blocks with a part each, in
    the 2-SM form (d = 10) and one CTA a unit (d = 200: the split form's rows do not
    stay resident)."""
    g = np.random.default_rng(d)
    for n in (100, 256, 257, 1025, 1100, 2049, 2300, 3400, 4500, 9100):
        x = g.normal(size=(n, d)).astype(np.float32)
        plain = hm.exact_knn(x, d, 9, "euclidean", "plain")
        knn = hm.exact_knn(x, d, 9, "euclidean", path)
        assert_same_bytes(knn.indices, plain.indices, f"{n} indices")
        assert_same_bytes(knn.dists, plain.dists, f"{n} dists")


@pytest.mark.parametrize("d,n,k,metric", [(64, 20000, 15, "cosine"), (300, 45000, 15, "euclidean")])
def test_clustered_rows_do_not_overflow_their_lists(d, n, k, metric):
    """Gaussian clusters whose rows have several hundred candidates, few of them far
    apart: the candidate lists of a single job hold them (a row that overflows costs an
    exact search of all of the points)."""
    import torch
    from holomap_b200.device import DeviceKnnProblem
    from holomap_b200.synth import serve_pool
    x = torch.from_numpy(np.ascontiguousarray(serve_pool(d, 0)[:n])).cuda()
    p = DeviceKnnProblem(n, d, k, metric, "auto")
    p.run(x)
    torch.cuda.synchronize()
    assert p.stats().overflow_rows == 0


@pytest.mark.parametrize("path", ["screen_bf16", "screen_bf16x3"])
@pytest.mark.parametrize("n,centres,k", [(6000, 1, 15), (6000, 14, 15), (20000, 31, 64), (20000, 33, 64), (20000, 60, 64)])
def test_fallback_rows_shared_by_columns(path, n, centres, k):
    """A few rows whose neighbours all lie at one distance (centres of a sphere of points)
    overflow their lists and take the exact search, several CTAs to a group of 32 rows:
    one group and two, one row and one short of a group, k of one list and of two."""
    import torch
    from holomap_b200.device import DeviceKnnProblem
    g = np.random.default_rng(n + centres)
    d = 48
    x = g.normal(size=(n, d))
    x /= np.linalg.norm(x, axis=1, keepdims=True)  # (the radii differ by the points' rounding)
    x[g.permutation(n)[:centres]] = 1e-6 * g.normal(size=(centres, d))
    x = torch.from_numpy(x.astype(np.float32)).cuda()
    want = DeviceKnnProblem(n, d, k, "euclidean", "plain")
    want.run(x)
    p = DeviceKnnProblem(n, d, k, "euclidean", path)
    for _ in range(2):  # (the second run finds the first one's counters)
        p.idx.fill_(-1)
        p.run(x)
        torch.cuda.synchronize()
        assert p.stats().overflow_rows >= centres
        assert torch.equal(p.idx, want.idx) and torch.equal(p.dist, want.dist)


@pytest.mark.parametrize("tight", [4000, 8200])  # 125 row groups: 3 CTAs each; 257: one each
def test_fallback_rows_of_a_tight_cluster(tight):
    """Thousands of rows in a cluster tighter than the screen's rounding, all of them
    searched exactly; as one job and in a batch of three."""
    import torch
    from holomap_b200.device import DeviceBatch, DeviceKnnProblem
    g = np.random.default_rng(tight)
    n, d, k = tight + 800, 24, 20
    x = g.normal(size=(n, d))
    x[g.permutation(n)[:tight]] *= 1e-4
    x = torch.from_numpy(x.astype(np.float32)).cuda()
    want = DeviceKnnProblem(n, d, k, "euclidean", "plain")
    want.run(x)
    p = DeviceKnnProblem(n, d, k, "euclidean", "screen_bf16")
    p.run(x)
    small = x[:500].contiguous()
    b = DeviceBatch([(small, k, "cosine", "screen_bf16"), (x, k, "euclidean", "screen_bf16"),
                     (small, 7, "euclidean", "screen_bf16")])
    b.run()
    torch.cuda.synchronize()
    assert p.stats().overflow_rows >= tight
    for idx, dist in ((p.idx, p.dist), b.problems[1][1:3]):
        assert torch.equal(idx, want.idx) and torch.equal(dist, want.dist)


@pytest.mark.parametrize("path", ["screen_bf16x3", "screen_tf32"])
@pytest.mark.parametrize("begin,end", [(1005, 1105), (7005, 7105), (11005, 11105)])
def test_rows_of_points_stored_cluster_by_cluster(path, begin, end):
    """A row's neighbours lie side by side, and its bound needs k chunks of the sample
    from its own cluster: with chunks of 64 columns the rows' lists overflowed."""
    import ctypes
    import torch
    from holomap_b200._lib import check as check_rc
    g = np.random.default_rng(3)
    n, d, k = 20000, 64, 15
    x = 4.0 * g.normal(size=(12, d))[np.sort(g.integers(0, 12, n))] + g.normal(size=(n, d))
    x = torch.from_numpy(x.astype(np.float32)).cuda()
    p = int(hm.KnnPath.parse(path))
    ws_bytes = hm.lib().hm_knn_rows_workspace_bytes(n, d, k, 0, p, begin, end)
    ws = torch.empty(ws_bytes + 256, dtype=torch.uint8, device="cuda")
    idx = torch.empty((end - begin) * k, dtype=torch.int32, device="cuda")
    dist = torch.empty((end - begin) * k, dtype=torch.float32, device="cuda")
    st = hm.HmStats()
    ptr = (ws.data_ptr() + 255) // 256 * 256
    check_rc(hm.lib().hm_knn_rows_device(x.data_ptr(), n, d, k, 0, p, begin, end, idx.data_ptr(), dist.data_ptr(),
                                         ptr, ws_bytes, None, ctypes.byref(st)))
    torch.cuda.synchronize()
    assert st.overflow_rows == 0
