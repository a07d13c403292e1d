"""All-pairs sums at the edges of how a call's sources are split over lanes, warps and
clusters, against FP64 (a term is evaluated to a few FP32 roundings and the sums are
compensated: 1e-6 of the summed magnitudes, as everywhere for brute force)."""
import numpy as np
import pytest

import oracle as O
import sbh_capi as C
import sbh_workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nq", [(1, 1), (31, 2), (127, 9), (128, 3), (129, 7), (1023, 1),
                                  (1024, 8), (4097, 65), (33333, 1), (33333, 130), (700, 20011)])
@pytest.mark.parametrize("dim,kernel", [(3, C.PLUMMER), (3, C.GRAVITY), (2, C.SMOOTH_DIST),
                                        (3, C.WINDING_NUMBER)])
def test_split_sums_match_fp64(n, nq, dim, kernel):
    pts, nrm, m = W.gaussian_mixture(n, seed=n, dim=dim)
    lo, hi = W.padded_box(pts)
    gpu = C.GpuTree(C.HostTree(pts, nrm, m, lo, hi, alpha=3.0))
    q = W.uniform_queries(nq, seed=nq, dim=dim, lo=-1.2, hi=1.2)
    v, _, c = gpu.eval(q, C.params(method=C.BRUTE_FORCE, kernel=kernel), contribs=True)
    k = slice(0, 400)
    ref = O.brute_force_f64(pts, nrm, m, kernel, q[k], alpha=3.0)
    scale = O.brute_force_f64(pts, nrm, m, kernel, q[k], alpha=3.0, abs_sum=True)
    assert (np.abs(v[k] - ref) <= 1e-6 * scale).all()
    assert (c == n).all()
    one, _ = gpu.eval(q[nq - 1:], C.params(method=C.BRUTE_FORCE, kernel=kernel))
    ref = O.brute_force_f64(pts, nrm, m, kernel, q[nq - 1:], alpha=3.0)
    scale = O.brute_force_f64(pts, nrm, m, kernel, q[nq - 1:], alpha=3.0, abs_sum=True)
    assert abs(one[0] - ref[0]) <= 1e-6 * scale[0] and abs(v[-1] - ref[0]) <= 1e-6 * scale[0]


@pytest.mark.parametrize("dim", [2, 3])
def test_gravity_at_the_reciprocals_limits(dim):
    """Distances beyond the shared reciprocal's range, at a source, infinite and NaN."""
    rng = np.random.default_rng(6)
    pts = rng.uniform(-1, 1, (515, dim)).astype(np.float32)
    m = rng.uniform(-1, 1, 515).astype(np.float32)
    lo, hi = W.padded_box(pts)
    gpu = C.GpuTree(C.HostTree(pts, np.ones_like(pts), m, lo, hi))
    q = np.array([[x] + [0.5] * (dim - 1) for x in
                  (0.1, 9e8, 2e9, 1e15, 1.5e19, 3e19, 1e30, np.inf, np.nan)], np.float32)
    q = np.concatenate([pts[7:8], q])
    v, _ = gpu.eval(q, C.params(method=C.BRUTE_FORCE, kernel=C.GRAVITY))
    scale = O.brute_force_f64(pts, np.ones_like(pts), m, C.GRAVITY, q[:6], abs_sum=True)
    ref = O.brute_force_f64(pts, np.ones_like(pts), m, C.GRAVITY, q[:6])
    assert (np.abs(v[:6] - ref) <= 1e-6 * scale).all()
    assert (v[6:9] == 0).all() and np.isnan(v[9])  # r^2 overflows: terms of m / inf
