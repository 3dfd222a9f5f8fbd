"""Performance cases: the work a user of this library has it do.

A user embeds datasets with holomap.  Every dataset goes through exact kNN and
smooth-kNN; a whole fit goes on to the fuzzy graph and its smallest
eigenpairs.  Programs that keep their points on the GPU use the device entry
points (``DeviceKnnProblem``, ``DeviceBatch``, the ``hm_*_device`` calls);
programs that hold numpy arrays use the drop-in calls ``knn_smooth``,
``fuzzy_simplicial_set`` and ``smallest_eigenpairs``.  The listed cases cover
both, from 1,000 points to 50,000, with the shapes, metrics and neighbour
counts of this repository's benchmark workloads and of its serving mix, ragged
sizes among them; ``draw`` gives other sizes of the same ranges.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import holomap_b200 as hm
from holomap_b200._lib import check, lib
from holomap_b200.device import DeviceBatch, DeviceKnnProblem

DEVICE = "cuda"


# ------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest everyday call: a notebook-sized dataset, latency-bound
        {"name": "knn_1k", "kind": "knn", "n": 1000, "d": 50, "k": 15, "metric": "euclidean", "data": "blobs"},
        # an ordinary serving request, ragged, clustered data under cosine
        {"name": "knn_5k_cosine", "kind": "knn", "n": 5003, "d": 300, "k": 15, "metric": "cosine",
         "data": "mixture"},
        # a mid-sized dataset with exact and one-ulp duplicates
        {"name": "knn_20k", "kind": "knn", "n": 20000, "d": 128, "k": 15, "metric": "euclidean", "data": "dups"},
        # the headline: 50,000 text embeddings
        {"name": "knn_embed_50k", "kind": "knn", "n": 50000, "d": 384, "k": 30, "metric": "cosine",
         "data": "embedding"},
        # the third metric of the serving mix (every pair in binary64)
        {"name": "knn_12k_manhattan", "kind": "knn", "n": 12007, "d": 64, "k": 15, "metric": "manhattan",
         "data": "mixture"},
        # many neighbours, as users ask for when they want global structure
        {"name": "knn_10k_k100", "kind": "knn", "n": 10000, "d": 32, "k": 100, "metric": "euclidean",
         "data": "mixture"},
        # many small datasets at once, replayed as one CUDA graph
        {"name": "batch_256", "kind": "batch", "count": 256, "n_lo": 200, "n_hi": 8000, "k": 15},
        # the drop-in call on host arrays
        {"name": "host_8k", "kind": "host_knn", "n": 8000, "d": 128, "k": 15, "metric": "euclidean",
         "data": "mixture"},
        # calibration of a gathered distance matrix, as row-sharded runs do it
        {"name": "smooth_150k", "kind": "smooth", "n": 150001, "k": 15},
        # the fuzzy graph of the headline's kNN graph
        {"name": "fuzzy_50k", "kind": "fuzzy", "n": 50000, "d": 384, "k": 30},
        # Laplacian and 3 smallest eigenpairs of that graph (a 2-d embedding's start)
        {"name": "spectral_50k", "kind": "spectral", "n": 50000, "d": 384, "k": 30, "pairs": 3},
        # a whole small fit up to the spectral layout, on host arrays
        {"name": "fit_2k", "kind": "fit", "n": 2000, "d": 50, "k": 15, "pairs": 3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["knn", "knn", "knn", "manhattan", "many", "batch", "host_knn", "smooth", "fuzzy", "spectral",
                       "fit"])
    if kind == "knn":
        n, d, k = _log_int(rng, 500, 50000), _log_int(rng, 16, 384), rng.randint(10, 30)
        metric = rng.choice(["euclidean", "cosine"])
        data = rng.choice(["mixture", "dups"] if metric == "euclidean" else ["mixture", "embedding"])
        return {"kind": "knn", "n": n, "d": d, "k": k, "metric": metric, "data": data}
    if kind == "manhattan":
        return {"kind": "knn", "n": _log_int(rng, 500, 13000), "d": _log_int(rng, 16, 128), "k": rng.randint(10, 30),
                "metric": "manhattan", "data": "mixture"}
    if kind == "many":
        return {"kind": "knn", "n": _log_int(rng, 1000, 12000), "d": _log_int(rng, 16, 64), "k": rng.randint(65, 150),
                "metric": rng.choice(["euclidean", "cosine"]), "data": "mixture"}
    if kind == "batch":
        return {"kind": "batch", "count": _log_int(rng, 16, 256), "n_lo": 200, "n_hi": _log_int(rng, 1000, 8000),
                "k": rng.randint(10, 30)}
    if kind == "host_knn":
        return {"kind": "host_knn", "n": _log_int(rng, 500, 16000), "d": _log_int(rng, 16, 300),
                "k": rng.randint(10, 30), "metric": rng.choice(["euclidean", "cosine"]), "data": "mixture"}
    if kind == "smooth":
        return {"kind": "smooth", "n": _log_int(rng, 2000, 250000), "k": rng.randint(10, 30)}
    if kind == "fuzzy":
        return {"kind": "fuzzy", "n": _log_int(rng, 2000, 50000), "d": rng.choice([64, 128, 384]),
                "k": rng.randint(10, 30)}
    if kind == "spectral":
        return {"kind": "spectral", "n": _log_int(rng, 3000, 50000), "d": rng.choice([64, 128, 384]),
                "k": rng.randint(10, 30), "pairs": rng.choice([3, 4])}
    return {"kind": "fit", "n": _log_int(rng, 500, 4000), "d": _log_int(rng, 16, 128), "k": rng.randint(10, 20),
            "pairs": 3}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    return g


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device=DEVICE, dtype=torch.float32)


def _uniform(g, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(*shape, generator=g, device=DEVICE, dtype=torch.float32)


def _mixture(g, n, d, clusters, centres, sigma_lo, sigma_hi):
    sigma = _uniform(g, sigma_lo, sigma_hi, clusters)
    labels = torch.randint(0, clusters, (n,), generator=g, device=DEVICE)
    return centres[labels] + _normal(g, n, d) * sigma[labels, None]


def _points(g, n, d, data):
    """n x d float32 points, as the repository's synthetic workloads shape them."""
    if data == "blobs":  # ten unit clusters around uniform centres
        return _mixture(g, n, d, 10, _uniform(g, -10.0, 10.0, 10, d), 1.0, 1.0).contiguous()
    if data == "embedding":  # a decaying spectrum, a shared offset, unit rows
        lam = torch.arange(1, d + 1, device=DEVICE, dtype=torch.float32) ** -0.6
        off = _normal(g, d)
        x = _normal(g, n, d) * lam + 0.3 * off / off.norm()
        return (x / x.norm(dim=1, keepdim=True)).contiguous()
    if data == "dups":  # 50 clusters; 5% exact copies, 2% copies one ulp away
        x = _mixture(g, n, d, 50, 4.0 * _normal(g, 50, d), 0.5, 2.0)
        perm = torch.randperm(n, generator=g, device=DEVICE)
        a, b = n // 20, n // 20 + n // 50
        src = perm[b:][torch.randint(0, n - b, (b,), generator=g, device=DEVICE)]
        x[perm[:b]] = x[src]
        col = torch.randint(0, d, (b - a,), generator=g, device=DEVICE)
        x[perm[a:b], col] = torch.nextafter(x[perm[a:b], col], torch.full((), math.inf, device=DEVICE))
        return x.contiguous()
    return _mixture(g, n, d, 12, 4.0 * _normal(g, 12, d), 0.3, 3.0).contiguous()


def _batch_points(case, seed):
    g = _gen(seed)
    r = np.random.Generator(np.random.PCG64(case["count"]))  # the sizes belong to the case
    out = []
    for _ in range(case["count"]):
        n = int(round(math.exp(r.uniform(math.log(case["n_lo"]), math.log(case["n_hi"])))))
        d = int(r.choice([16, 50, 128]))
        clusters = int(r.integers(3, 21))
        metric = "euclidean" if r.uniform() < 0.7 else "cosine"
        x = _mixture(g, n, d, clusters, _uniform(g, -10.0, 10.0, clusters, d), 0.3, 3.0).contiguous()
        out.append((x, case["k"], metric))
    return out


def _smooth_dists(case, seed):
    """n x k ascending distances, self first, of the sizes kNN graphs have; a
    few rows start with exact duplicates."""
    g = _gen(seed)
    n, k = case["n"], case["k"]
    base = _uniform(g, 0.2, 4.0, n, 1)
    steps = _uniform(g, 0.0, 0.1, n, k) * base
    d = base + torch.cumsum(steps, 1) - steps
    d[:, 0] = 0.0
    d[::97, 1] = 0.0
    return d.contiguous()


def _knn_graph(x, k):
    p = DeviceKnnProblem(x.shape[0], x.shape[1], k, "cosine")
    p.run(x)
    return p


class _Fuzzy:
    """Buffers of one hm_fuzzy_graph_device problem."""

    def __init__(self, n, k):
        cap = 2 * n * k
        self.rows = torch.zeros(cap, dtype=torch.int32, device=DEVICE)
        self.cols = torch.zeros(cap, dtype=torch.int32, device=DEVICE)
        self.vals = torch.zeros(cap, dtype=torch.float32, device=DEVICE)
        self.nnz = torch.zeros(1, dtype=torch.int64, device=DEVICE)
        self.ws_bytes = lib().hm_fuzzy_workspace_bytes(n, k)
        self.ws = torch.empty(self.ws_bytes + 256, dtype=torch.uint8, device=DEVICE)
        self.ws_ptr = (self.ws.data_ptr() + 255) // 256 * 256

    def run(self, idx, dist, sigma, rho, n, k):
        check(lib().hm_fuzzy_graph_device(
            idx.data_ptr(), dist.data_ptr(), sigma.data_ptr(), rho.data_ptr(), n, k, self.rows.data_ptr(),
            self.cols.data_ptr(), self.vals.data_ptr(), self.nnz.data_ptr(), self.ws_ptr, self.ws_bytes,
            torch.cuda.current_stream().cuda_stream))


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "knn":
        st["x"] = _points(_gen(seed), case["n"], case["d"], case["data"])
        st["problem"] = DeviceKnnProblem(case["n"], case["d"], case["k"], case["metric"])
    elif kind == "batch":
        st["batch"] = DeviceBatch(_batch_points(case, seed))
    elif kind == "host_knn":
        st["x"] = _points(_gen(seed), case["n"], case["d"], case["data"]).cpu().numpy()
    elif kind == "smooth":
        n = case["n"]
        st["dist"] = _smooth_dists(case, seed)
        st["sigma"] = torch.empty(n, dtype=torch.float32, device=DEVICE)
        st["rho"] = torch.empty(n, dtype=torch.float32, device=DEVICE)
        st["ws"] = torch.empty(lib().hm_smooth_workspace_bytes(n) + 256, dtype=torch.uint8, device=DEVICE)
        st["ws_ptr"] = (st["ws"].data_ptr() + 255) // 256 * 256
    elif kind in ("fuzzy", "spectral"):
        n, k = case["n"], case["k"]
        p = _knn_graph(_points(_gen(seed), n, case["d"], "embedding"), k)
        f = _Fuzzy(n, k)
        if kind == "fuzzy":
            st["graph"] = (p.idx, p.dist, p.sigma, p.rho)
            st["fuzzy"] = f
        else:
            f.run(p.idx, p.dist, p.sigma, p.rho, n, k)
            nnz = int(f.nnz.item())
            st["coo"] = tuple(t[:nnz].clone() for t in (f.rows, f.cols, f.vals))
            st["indptr"] = torch.empty(n + 1, dtype=torch.int64, device=DEVICE)
            st["svals"] = torch.zeros(2 * n * k, dtype=torch.float64, device=DEVICE)
            st["degrees"] = torch.empty(n, dtype=torch.float64, device=DEVICE)
            st["ws_bytes"] = lib().hm_eigenpairs_workspace_bytes(n, case["pairs"])
            st["ws"] = torch.empty(st["ws_bytes"] + 256, dtype=torch.uint8, device=DEVICE)
            st["ws_ptr"] = (st["ws"].data_ptr() + 255) // 256 * 256
            st["values"] = np.zeros(case["pairs"])
            st["vectors"] = np.zeros((case["pairs"], n))
    else:  # fit
        st["x"] = _points(_gen(seed), case["n"], case["d"], "embedding").cpu().numpy()
    return st


# --------------------------------------------------------------- one pass
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "knn":
        p = st["problem"]
        p.run(st["x"])
        return {"idx": p.idx, "dist": p.dist, "sigma": p.sigma, "rho": p.rho}
    if kind == "batch":
        st["batch"].run(graph=True)
        return st["batch"].out.view(torch.int32)  # indices and float bits of every dataset
    if kind == "host_knn":
        knn, sm = hm.knn_smooth(st["x"], case["d"], case["k"], case["metric"])
        return {"idx": knn.indices, "dist": knn.dists, "sigma": sm.sigmas, "rho": sm.rhos}
    if kind == "smooth":
        check(lib().hm_smooth_knn_device(st["dist"].data_ptr(), case["n"], case["k"], st["sigma"].data_ptr(),
                                         st["rho"].data_ptr(), st["ws_ptr"],
                                         torch.cuda.current_stream().cuda_stream))
        return {"sigma": st["sigma"], "rho": st["rho"]}
    if kind == "fuzzy":
        f = st["fuzzy"]
        f.run(*st["graph"], case["n"], case["k"])
        return {"rows": f.rows, "cols": f.cols, "vals": f.vals, "nnz": f.nnz}
    if kind == "spectral":
        rows, cols, vals = st["coo"]
        n, s = case["n"], torch.cuda.current_stream().cuda_stream
        check(lib().hm_laplacian_device(rows.data_ptr(), cols.data_ptr(), vals.data_ptr(), n, rows.numel(),
                                        st["indptr"].data_ptr(), st["svals"].data_ptr(), st["degrees"].data_ptr(), s))
        found, cycles = ctypes.c_uint32(0), ctypes.c_uint32(0)
        check(lib().hm_eigenpairs_device(st["indptr"].data_ptr(), cols.data_ptr(), st["svals"].data_ptr(), n,
                                         case["pairs"], st["ws_ptr"], st["ws_bytes"], s, st["values"].ctypes.data,
                                         st["vectors"].ctypes.data, ctypes.byref(found), ctypes.byref(cycles)))
        return {"indptr": st["indptr"], "svals": st["svals"], "degrees": st["degrees"], "values": st["values"],
                "vectors": st["vectors"]}
    knn, sm = hm.knn_smooth(st["x"], case["d"], case["k"], "cosine")
    g = hm.fuzzy_simplicial_set(knn, sm)
    e = hm.smallest_eigenpairs(g, case["pairs"])
    return {"idx": knn.indices, "dist": knn.dists, "sigma": sm.sigmas, "rho": sm.rhos, "values": e.values,
            "vectors": e.vectors}


# -------------------------------------------------- what a pass cannot avoid
def work(case):
    kind = case["kind"]

    def knn(n, d, k):  # points in; indices, distances, sigma, rho out; every pair once
        return 4 * n * d + 8 * n * k + 8 * n, 2 * n * n * d

    if kind in ("knn", "host_knn"):
        b, f = knn(case["n"], case["d"], case["k"])
        return {"bytes": b, "flops": f}
    if kind == "batch":
        lo, hi, c = case["n_lo"], case["n_hi"], case["count"]
        ln = math.log(hi / lo)
        n1, n2 = (hi - lo) / ln, (hi * hi - lo * lo) / (2 * ln)  # means of n and n^2
        d = (16 + 50 + 128) / 3
        return {"bytes": c * n1 * (4 * d + 8 * case["k"] + 8), "flops": c * 2 * n2 * d}
    if kind == "smooth":
        return {"bytes": 4 * case["n"] * case["k"] + 8 * case["n"], "flops": 0}
    n, k = case["n"], case["k"]
    nnz = 1.7 * n * k  # a kNN graph's union is about 1.7 entries per directed edge
    if kind == "fuzzy":
        return {"bytes": 8 * n * k + 8 * n + 12 * nnz, "flops": 0}
    # Laplacian: COO in, offsets, weights and degrees out; one Lanczos cycle of
    # 60 steps over it and the vectors out
    steps, m = max(8 * case["pairs"], 60), case["pairs"]
    spectral = (12 * nnz + 8 * nnz + 24 * n + 8 * n * m, 2 * nnz * steps + 4 * n * steps * steps)
    if kind == "spectral":
        return {"bytes": spectral[0], "flops": spectral[1]}
    b, f = knn(n, case["d"], k)
    return {"bytes": b + 12 * nnz + spectral[0], "flops": f + spectral[1]}


# ----------------------------------------------------- 64-bit results
def _exact_dists(x, k, metric):
    """(n x k ascending distances, their columns) in float64."""
    x = x.double()
    n = x.shape[0]
    out, cols = [], []
    norm = (x * x).sum(1)
    unit = x / x.norm(dim=1, keepdim=True).clamp_min(1e-300)
    step = max(1, min(n, (1 << 27) // n))
    take = min(n, k + 8)
    for a in range(0, n, step):
        b = min(n, a + step)
        if metric == "manhattan":
            c = torch.cdist(x[a:b], x, p=1)
        elif metric == "cosine":
            c = (1.0 - unit[a:b] @ unit.T).clamp_min(0.0)
        else:
            c = norm[a:b, None] + norm[None, :] - 2.0 * (x[a:b] @ x.T)
        c[torch.arange(b - a, device=x.device), torch.arange(a, b, device=x.device)] = -1.0  # self
        c, j = c.topk(take, 1, largest=False, sorted=True)
        if metric == "euclidean":  # the differences themselves, without cancellation
            c = torch.cat([(x[a + q:min(a + q + 256, b), None, :] - x[j[q:q + 256]]).square().sum(2).sqrt()
                           for q in range(0, b - a, 256)])
        c[j == torch.arange(a, b, device=x.device)[:, None]] = 0.0
        c, o = torch.sort(c, dim=1, stable=True)
        out.append(c[:, :k])
        cols.append(j.gather(1, o)[:, :k])
    return torch.cat(out), torch.cat(cols)


def _exact_smooth(d):
    """(sigma, rho) of ascending float64 distances."""
    n, k = d.shape
    target = math.log2(k)
    pos = d > 0
    rho = torch.where(pos.any(1), d.gather(1, pos.int().argmax(1, keepdim=True))[:, 0], torch.zeros_like(d[:, 0]))
    gap = (d[:, 1:] - rho[:, None]).clamp_min(0.0)
    big = 3.4028234663852886e38
    lo, hi, mid = torch.zeros(n).to(d), torch.full((n,), big).to(d), torch.ones(n).to(d)
    open_ = torch.ones(n, dtype=torch.bool, device=d.device)
    for _ in range(64):
        psum = torch.exp(-gap / mid[:, None]).sum(1)
        open_ = open_ & ((psum - target).abs() >= 1e-5)
        over = psum > target
        hi2, lo2 = torch.where(over, mid, hi), torch.where(over, lo, mid)
        new = torch.where(~over & (hi2 >= big), mid * 2.0, (lo2 + hi2) / 2.0)
        lo, hi, mid = (torch.where(open_, q, p) for q, p in ((lo2, lo), (hi2, hi), (new, mid)))
    floor = torch.where(rho > 0, d.mean(1), d.mean().expand(n)) * 1e-3
    return torch.maximum(mid, floor), rho


def _exact_fuzzy(idx, dist, sigma, rho, n, k):
    """(row * n + col keys ascending, float64 strengths) of the symmetric graph."""
    r = torch.arange(n, device=idx.device).repeat_interleave(k)
    c = idx.reshape(-1).long()
    gap = dist.double().reshape(-1) - rho.double()[r]
    sg = sigma.double()[r]
    v = torch.where((gap <= 0) | (sg == 0), torch.ones_like(gap), torch.exp(-gap / sg))
    keep = (c != r) & (v > 0)
    r, c, v = r[keep], c[keep], v[keep]
    key, inv = torch.unique(torch.cat([r * n + c, c * n + r]), return_inverse=True)
    one = torch.zeros(key.numel(), dtype=torch.float64, device=key.device)
    two = one.clone()
    one[inv[:r.numel()]] = v
    two[inv[r.numel():]] = v
    return key, one + two - one * two


def _exact_eigen(rows, cols, vals, n, pairs):
    """(values, vectors as rows) of the dense normalized Laplacian."""
    w = torch.zeros(n, n, dtype=torch.float64, device=vals.device)
    w[rows, cols] = vals.double()
    s = w.sum(1).rsqrt()
    lam, vec = torch.linalg.eigh(torch.eye(n, dtype=torch.float64, device=w.device) - s[:, None] * w * s[None, :])
    lam, vec = lam[:pairs], vec[:, :pairs].T.contiguous()
    at = (vec.abs() > vec.abs().amax(1, keepdim=True) - 1e-12).int().argmax(1, keepdim=True)
    return lam, vec * vec.gather(1, at).sign()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("knn", "host_knn"):
        x = _points(_gen(seed), case["n"], case["d"], case["data"])
        dist, _ = _exact_dists(x, case["k"], case["metric"])
        sigma, rho = _exact_smooth(dist)
        return {"idx": None, "dist": dist.reshape(-1), "sigma": sigma, "rho": rho}
    if kind == "smooth":
        sigma, rho = _exact_smooth(_smooth_dists(case, seed).double())
        return {"sigma": sigma, "rho": rho}
    if kind == "fuzzy":
        st = prepare(case, seed)  # its inputs are a kNN graph of this library
        n, k = case["n"], case["k"]
        _, v = _exact_fuzzy(st["graph"][0], *st["graph"][1:], n, k)
        vals = torch.zeros(2 * n * k, dtype=torch.float64, device=DEVICE)
        vals[:v.numel()] = v
        return {"rows": None, "cols": None, "vals": vals, "nnz": None}
    if kind == "spectral":
        st = prepare(case, seed)  # its input is a fuzzy graph of this library
        rows, cols, vals = st["coo"]
        n, rows, cols = case["n"], rows.long(), cols.long()
        deg = torch.zeros(n, dtype=torch.float64, device=DEVICE).index_add_(0, rows, vals.double())
        s = torch.zeros(2 * n * case["k"], dtype=torch.float64, device=DEVICE)
        s[:rows.numel()] = vals.double() * deg.rsqrt()[rows] * deg.rsqrt()[cols]
        values = vectors = None
        if n <= 8000:
            values, vectors = _exact_eigen(rows, cols, vals, n, case["pairs"])
        return {"indptr": None, "svals": s, "degrees": deg, "values": values, "vectors": vectors}
    if kind == "fit":
        x = _points(_gen(seed), case["n"], case["d"], "embedding")
        n, k = case["n"], case["k"]
        dist, idx = _exact_dists(x, k, "cosine")
        sigma, rho = _exact_smooth(dist)
        key, v = _exact_fuzzy(idx, dist, sigma, rho, n, k)
        values, vectors = _exact_eigen(key // n, key % n, v, n, case["pairs"])
        return {"idx": None, "dist": dist.reshape(-1), "sigma": sigma, "rho": rho, "values": values,
                "vectors": vectors}
    return None
