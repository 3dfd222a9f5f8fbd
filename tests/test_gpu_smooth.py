"""smooth-kNN alone (hm_smooth_knn) against the oracle, byte for byte, where the
calibration kernel's row widths, lane counts and bracketed bisection have their
edges: k around the widths 16, 32, 64, 128 and 256, row counts around the
changes of lanes per row, and rows for which the bracket has one side or none
(ties with rho, all gaps zero, infinite gaps, gaps far from 1, unsorted rows)."""
import numpy as np
import pytest

import holomap_b200 as hm
from parity import assert_same_bytes

pytestmark = pytest.mark.gpu


def rows_of(kind, n, k, seed=5):
    g = np.random.default_rng(seed)
    if kind == "graph":  # ascending distances of a kNN graph's shape, some duplicates
        base = g.uniform(0.2, 4.0, (n, 1))
        d = base + np.cumsum(g.uniform(0.0, 0.1, (n, k)) * base, 1)
        d[:, 0] = 0.0
        if k > 1:
            d[::97, 1] = 0.0
    elif kind == "grid":  # many ties and zero gaps
        d = np.sort(np.floor(g.uniform(0.0, 4.0, (n, k))), 1)
    elif kind == "ties":  # 1 .. k - 1 entries tied with rho
        d = np.sort(g.uniform(1.0, 2.0, (n, k)), 1)
        z = g.integers(1, max(2, k), (n, 1))
        d[(np.arange(k)[None, :] >= 1) & (np.arange(k)[None, :] <= z)] = 1.0
        d[:, 0] = 0.0
    elif kind == "wide":
        d = np.sort(np.exp(g.normal(0.0, 8.0, (n, k))), 1)
    elif kind == "tiny":
        d = np.sort(g.uniform(0.0, 1e-42, (n, k)), 1)
    elif kind == "inf":
        d = np.sort(g.uniform(0.0, 1.0, (n, k)), 1)
        d[::3, -1] = np.inf
        d[::7, -2:] = np.inf
    else:  # "unsorted", negative values among them
        d = g.normal(0.0, 1.0, (n, k))
    return np.ascontiguousarray(d.astype(np.float32))


def check(oracle, d, k, what):
    sm = hm.smooth_knn(d, k)
    osig, orho = oracle.smooth_knn(d, k)
    assert_same_bytes(sm.rhos, orho, f"{what} rho")
    assert_same_bytes(sm.sigmas, osig, f"{what} sigma")


@pytest.mark.parametrize("k", [1, 2, 3, 5, 15, 16, 17, 31, 32, 33, 64, 65, 128, 129, 256, 257])
@pytest.mark.parametrize("kind", ["graph", "grid", "ties", "wide", "tiny", "inf", "unsorted"])
def test_row_widths(oracle, kind, k):
    check(oracle, rows_of(kind, 131, k), k, f"{kind} k={k}")


@pytest.mark.parametrize("n,k", [(1, 15), (16383, 16), (16384, 12), (16384, 30), (32767, 9), (32768, 16)])
def test_row_counts(oracle, n, k):
    check(oracle, rows_of("graph", n, k), k, f"n={n} k={k}")
