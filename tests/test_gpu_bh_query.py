"""Barnes-Hut calls small enough to run a warp per query against calls that run a
lane per query: the same nodes opened and the same sums, bit for bit."""
import numpy as np
import pytest

import sbh_capi as C
import sbh_workloads as W
from helpers import bits_equal

pytestmark = pytest.mark.gpu


def _points(kind, dim):
    rng = np.random.default_rng(5)
    if kind == "one":
        pts = np.zeros((1, dim), np.float32)
    elif kind == "chain":  # pairs 1e-6 apart: chains of single-child nodes, many levels
        a = rng.uniform(-1, 1, (200, dim))
        pts = np.concatenate([a, a + 1e-6]).astype(np.float32)
    else:
        pts = W.gaussian_mixture(6000, seed=6, dim=dim)[0]
    n = len(pts)
    nrm = rng.normal(size=(n, dim)).astype(np.float32)
    return pts, nrm, rng.uniform(0.5, 1.5, n).astype(np.float32)


@pytest.mark.parametrize("kind,dim,dsl,leaf,kernel,beta", [
    ("gauss", 3, 1, 1, C.GRAVITY, 2.0), ("gauss", 3, 1, 8, C.PLUMMER, 2.0),
    ("gauss", 3, 2, 1, C.WINDING_NUMBER, 1.25), ("gauss", 3, 3, 33, C.GRAVITY, 5.0),
    ("gauss", 2, 1, 1, C.SMOOTH_DIST, 3.0), ("gauss", 2, 3, 4, C.WINDING_NUMBER, 2.0),
    ("gauss", 2, 1, 1, C.GRAVITY, 0.0), ("gauss", 3, 1, 2, C.GRAVITY, float("inf")),
    ("gauss", 2, 2, 1, C.PLUMMER, -1.0), ("gauss", 2, 2, 1, C.PLUMMER, 1e-30),
    ("chain", 3, 1, 1, C.GRAVITY, 50.0), ("chain", 2, 1, 1, C.GRAVITY, 2.0),
    ("one", 3, 2, 1, C.PLUMMER, 2.0), ("one", 2, 1, 4, C.GRAVITY, 2.0)])
def test_query_walk_equals_lane_walk(kind, dim, dsl, leaf, kernel, beta):
    torch = pytest.importorskip("torch")
    pts, nrm, m = _points(kind, dim)
    lo, hi = W.padded_box(pts)
    gpu = C.GpuTree(C.HostTree(pts, nrm, m, lo, hi, alpha=3.0, dim_split_log=dsl, leaf_size=leaf))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    small = 3001
    q = np.random.default_rng(7).uniform(-1.5, 1.5, (small, dim)).astype(np.float32)
    q[:4] = [[0] * dim, pts[0], [np.nan] * dim, [1e25] * dim]
    p = C.params(method=C.BARNES_HUT, kernel=kernel, beta=beta)
    v, _, c = gpu.eval(q, p, contribs=True)
    # the lane walk needs over 2,048 queries per SM: the same queries, then copies of one
    big = np.concatenate([q, np.repeat(q[-1:], 2048 * sms + 1 - small, axis=0)])
    bv, _, bc = gpu.eval(big, p, contribs=True)
    nan = np.isnan(bv[:small])
    assert np.array_equal(np.isnan(v), nan) and bits_equal(v[~nan], bv[:small][~nan])
    assert np.array_equal(c, bc[:small])
    # one query at a time, and with the ordering that larger calls of this kind use
    one, _, oc = gpu.eval(q[5:6], p, contribs=True)
    assert bits_equal(one, v[5:6]) and oc[0] == c[5]
    mid = np.concatenate([q, np.repeat(q[-1:], 20000 - small, axis=0)])
    assert bits_equal(gpu.eval(mid, p)[0][:small][~nan], v[~nan])
