"""Smooth-distance gradients with NaN inputs: the value and the gradient are NaN, wherever in the
sums the NaN comes and whichever kernel forms them; other queries of the call keep their bits."""
import numpy as np
import pytest

import sbh_capi as C
import sbh_workloads as W
from helpers import bits_equal

pytestmark = pytest.mark.gpu
NAN = float("nan")


def _tree(pts, n, dim, **kw):
    nrm, m = np.ones((n, dim), np.float32), np.ones(n, np.float32)
    return C.GpuTree(C.HostTree(pts, nrm, m, np.full(dim, -1.5, np.float32),
                                np.full(dim, 1.5, np.float32), alpha=20.0, **kw))


@pytest.mark.parametrize("n", [1, 4, 128, 129, 5000])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("method", [C.BRUTE_FORCE, C.BARNES_HUT, C.BARNES_HUT_VOTE, C.STOCHASTIC])
def test_nan_query(n, dim, method):
    if method == C.STOCHASTIC and n == 1:
        pytest.skip("a one-leaf tree has no subdomains: every estimate is 0")
    pts = np.random.default_rng(n).uniform(-1, 1, (n, dim)).astype(np.float32)
    gpu = _tree(pts, n, dim, dim_split_log=2)
    q = W.uniform_queries(70, seed=1, dim=dim)
    # KEEP_ORDER and beta = inf: the company of a vote changes nothing
    p = C.params(method=method, kernel=C.SMOOTH_DIST, beta=float("inf"), seed=3)
    v, g, _ = gpu.eval_grad(q, p)
    for k, d in ((0, 0), (33, dim - 1), (69, 1)):
        b = q.copy()
        b[k, d] = NAN
        bv, bg, _ = gpu.eval_grad(b, p)
        assert np.isnan(bv[k]) and np.isnan(bg[k]).all()
        rest = np.arange(70) != k
        if method != C.BRUTE_FORCE:
            assert bits_equal(bv[rest], v[rest])
            assert bits_equal(np.ascontiguousarray(bg[rest]), np.ascontiguousarray(g[rest]))
        else:  # a pair's other query may have its group summed term by term
            assert np.all(np.abs(bv[rest] - v[rest]) <= 1e-5 * np.abs(v[rest]) + 1e-6)


@pytest.mark.parametrize("n", [1, 4, 128, 129, 300, 5000])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("at", ["first", "later"])
@pytest.mark.parametrize("method", [C.BRUTE_FORCE, C.BARNES_HUT])
def test_nan_source(n, dim, at, method):
    pts = np.random.default_rng(n).uniform(-1, 1, (n, dim)).astype(np.float32)
    k = n // 2
    pts[k] = NAN if at == "first" else 0.9  # first cell of every node, or of its own row
    pts[k, 0] = NAN
    gpu = _tree(pts, n, dim)
    for nq in (1, 40):
        v, g, _ = gpu.eval_grad(W.uniform_queries(nq, seed=2, dim=dim),
                                C.params(method=method, kernel=C.SMOOTH_DIST, beta=2.0))
        assert np.isnan(v).all() and np.isnan(g).all()
