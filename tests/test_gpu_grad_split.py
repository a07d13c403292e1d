"""All-pairs gradients at the edges of the source split, at sources and at distances whose
square is an FP32 subnormal, against FP64 (tolerances of test_gpu_grad.py)."""
import numpy as np
import pytest

import oracle as O
import sbh_capi as C
import sbh_workloads as W

pytestmark = pytest.mark.gpu
ALPHA = 25.0


@pytest.mark.parametrize("n,nq", [(1, 5), (31, 6), (127, 9), (128, 7), (129, 8), (1024, 12),
                                  (4097, 70), (20000, 5), (700, 9001)])
@pytest.mark.parametrize("dim,kernel", [(2, C.GRAVITY), (3, C.PLUMMER), (2, C.SMOOTH_DIST),
                                        (3, C.SMOOTH_DIST), (3, C.GRAVITY)])
def test_split_gradients_match_fp64(n, nq, dim, kernel):
    pts, nrm, m = W.gaussian_mixture(n, seed=n, dim=dim)
    pts[0] = 0.0
    lo, hi = W.padded_box(pts)
    gpu = C.GpuTree(C.HostTree(pts, nrm, m, lo - 1, hi + 1, alpha=ALPHA))
    q = W.uniform_queries(nq, seed=nq, dim=dim, lo=-1.2, hi=1.2)
    q[0] = pts[n // 2]
    q[1] = [1e-20] + [0.0] * (dim - 1)
    q[2] = pts[n - 1]
    q[-1] = [40.0] * dim
    v, g, _, c = gpu.eval_grad(q, C.params(method=C.BRUTE_FORCE, kernel=kernel), contribs=True)
    keep = np.r_[0:min(nq, 300), nq - 1]
    ov, og = O.brute_force_grad_f64(pts, m, kernel, q[keep], ALPHA)
    # the oracle's own sum underflows FP64 at the far query; the product's must not
    assert np.isfinite(v).all() and np.isfinite(g).all()
    known = np.isfinite(og).all(axis=1)
    assert known[:min(nq, 300) - (nq <= 300)].all()
    keep, ov, og = keep[known], ov[known], og[known]
    floor = 1e-6 if kernel == C.SMOOTH_DIST else 0.0
    assert np.all(np.abs(v[keep] - ov) <= 1e-5 * np.abs(ov) + floor)
    err = np.linalg.norm(g[keep].astype(np.float64) - og, axis=1)
    assert np.all(err <= 1e-4 * np.linalg.norm(og, axis=1) + 1e-6)
    assert (c == n).all()
    v0, g0, _ = gpu.eval_grad(q[:1], C.params(method=C.BRUTE_FORCE, kernel=kernel))
    assert abs(v0[0] - ov[0]) <= 1e-5 * abs(ov[0]) + floor
    assert np.linalg.norm(g0[0] - og[0]) <= 1e-4 * np.linalg.norm(og[0]) + 1e-6
