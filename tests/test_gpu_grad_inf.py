"""Smooth-distance gradients by brute force with a source beyond every finite distance: its term
is e^-inf, so values and gradients are those of the other sources, wherever it comes in the sums."""
import numpy as np
import pytest

import oracle as O
import sbh_capi as C
import sbh_workloads as W

pytestmark = pytest.mark.gpu
ALPHA = 20.0


@pytest.mark.parametrize("n", [2, 33, 128, 129, 300, 5000])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("far", [float("inf"), float("-inf"), 1e25])
def test_far_source(n, dim, far):
    pts = np.random.default_rng(n).uniform(-1, 1, (n, dim)).astype(np.float32)
    pts[n // 2] = 0.9
    pts[n // 2, 0] = far
    box = np.full(dim, 1.5, np.float32)
    gpu = C.GpuTree(C.HostTree(pts, np.ones((n, dim), np.float32), np.ones(n, np.float32), -box,
                               box, alpha=ALPHA))
    rest = np.delete(pts, n // 2, axis=0)
    for nq in (1, 40):
        q = W.uniform_queries(nq, seed=2, dim=dim)
        v, g, _ = gpu.eval_grad(q, C.params(method=C.BRUTE_FORCE, kernel=C.SMOOTH_DIST))
        ov, og = O.brute_force_grad_f64(rest, np.ones(n - 1, np.float32), C.SMOOTH_DIST, q, ALPHA)
        # the bounds of test_gpu_grad.py's brute-force checks
        assert np.all(np.abs(v - ov) <= 1e-5 * np.abs(ov) + 1e-6)
        err = np.linalg.norm(g.astype(np.float64) - og, axis=1)
        assert np.all(err <= 1e-4 * np.linalg.norm(og, axis=1) + 1e-6)


@pytest.mark.parametrize("n", [1, 4, 128, 129])
@pytest.mark.parametrize("dim", [2, 3])
def test_no_source_in_reach(n, dim):
    """All terms are zero: the value is infinite, the gradient 0 / 0."""
    pts = np.full((n, dim), 1e25, np.float32)
    box = np.full(dim, 1.5, np.float32)
    gpu = C.GpuTree(C.HostTree(pts, np.ones((n, dim), np.float32), np.ones(n, np.float32), -box,
                               box, alpha=ALPHA, max_depth=3))
    v, g, _ = gpu.eval_grad(W.uniform_queries(3, seed=2, dim=dim),
                            C.params(method=C.BRUTE_FORCE, kernel=C.SMOOTH_DIST))
    assert np.all(v == np.inf) and np.isnan(g).all()
