"""Smooth-distance gradients by brute force where the first sources of every lane are far behind
the ones that count: the reference exponent of the sums must follow."""
import numpy as np
import pytest

import oracle as O
import sbh_capi as C
import sbh_workloads as W

pytestmark = pytest.mark.gpu
ALPHA = 25.0


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("lag", [0.5, 3.9, 8.0, 20.0, 39.0])
def test_far_sources_first(dim, lag):
    rng = np.random.default_rng(5)
    step = lag / ALPHA / np.sqrt(dim)

    def cloud(n, half, at):
        return rng.uniform(-half, half, (n, dim)) / ALPHA + at * step

    # in tree order: far sources, the four that count, far ones again
    pts = np.concatenate([cloud(24000, 0.02, 0), cloud(4, 0.5, 1),
                          cloud(8000, 0.02, 2)]).astype(np.float32)
    m = np.ones(len(pts), np.float32)
    gpu = C.GpuTree(C.HostTree(pts, np.ones_like(pts), m, *W.padded_box(pts), alpha=ALPHA))
    q = cloud(2000, 0.5, 1).astype(np.float32)
    v, g, _ = gpu.eval_grad(q, C.params(method=C.BRUTE_FORCE, kernel=C.SMOOTH_DIST))
    ov, og = O.brute_force_grad_f64(pts, m, C.SMOOTH_DIST, q, ALPHA)
    # A term's relative error: the exponent (up to about 2 in magnitude: the root 2^-23 and
    # the product 2^-24 of it, 4e-7), its difference and product with log2 e (up to 8: 4.8e-7 each,
    # times ln 2), the MUFU's power and root (2^-22 each): 1.5e-6 together, about a quarter of
    # it typically.  Gradients are means of unit vectors, so twice that at most.
    err = np.linalg.norm(g - og, axis=1)
    assert np.max(err) <= 3e-6 and np.median(err) <= 4e-7
    verr = np.abs(v - ov) * ALPHA
    assert np.max(verr) <= 2e-6 and np.median(verr) <= 4e-7
