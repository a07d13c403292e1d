"""The sampler's results do not depend on how many queries a warp takes (1 to 32 by the
call's size), which decides how its first level is summed: bit for bit."""
import numpy as np
import pytest

import sbh_capi as C
import sbh_workloads as W
from helpers import bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,dsl,leaf,kernel,grad", [
    (3, 2, 1, C.GRAVITY, False), (3, 1, 8, C.WINDING_NUMBER, False), (2, 2, 1, C.SMOOTH_DIST, False),
    (2, 1, 3, C.PLUMMER, False), (2, 2, 1, C.GRAVITY, True), (3, 1, 4, C.SMOOTH_DIST, True)])
def test_results_do_not_depend_on_the_group(dim, dsl, leaf, kernel, grad):
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    pts, nrm, m = W.gaussian_mixture(1500, seed=3, dim=dim)
    lo, hi = W.padded_box(pts)
    gpu = C.GpuTree(C.HostTree(pts, nrm, m, lo, hi, alpha=5.0, dim_split_log=dsl, leaf_size=leaf))
    # groups of 32 (the last one ragged), 16, 8, 4, 2 and 1
    sizes = [256 * 16 * sms + 77] + [128 * g * sms - 5 for g in (8, 4, 2, 1)] + [33, 1]
    q = np.random.default_rng(4).uniform(-1.3, 1.3, (sizes[0], dim)).astype(np.float32)
    p = C.params(method=C.STOCHASTIC, kernel=kernel, samples_per_subdomain=1, seed=9)

    def run(n):
        if grad:
            v, g, _, c = gpu.eval_grad(q[:n], p, contribs=True)
            return v, g, c
        v, _, c = gpu.eval(q[:n], p, contribs=True)
        return v, v, c

    v, g, c = run(sizes[0])
    for n in sizes[1:]:
        a, b, d = run(n)
        assert bits_equal(a, v[:n]) and bits_equal(np.ascontiguousarray(b), np.ascontiguousarray(g[:n]))
        assert np.array_equal(d, c[:n])
    # a ragged tail: the last warp of 32 holds 13 queries, and alone they are in warps of one
    a, b, d = run(sizes[0])
    assert bits_equal(a, v)
