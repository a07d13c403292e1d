"""The sampler with 16 queries a warp, the most whose first-level terms wait in shared memory, and
with ragged last warps: the same bits as in calls where the same queries fall into other warps."""
import numpy as np
import pytest

import sbh_capi as C
import sbh_workloads as W
from helpers import bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,dsl,leaf,kernel,grad", [
    (3, 2, 1, C.WINDING_NUMBER, False), (3, 1, 8, C.GRAVITY, False), (2, 3, 1, C.PLUMMER, False),
    (2, 1, 3, C.SMOOTH_DIST, False), (3, 2, 1, C.PLUMMER, True), (2, 2, 4, C.SMOOTH_DIST, True)])
def test_groups_of_16_and_tails(dim, dsl, leaf, kernel, grad):
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    pts, nrm, m = W.gaussian_mixture(1500, seed=6, dim=dim)
    lo, hi = W.padded_box(pts)
    gpu = C.GpuTree(C.HostTree(pts, nrm, m, lo, hi, alpha=5.0, dim_split_log=dsl, leaf_size=leaf))
    most = 256 * 16 * sms  # the largest call in warps of 16 queries
    q = np.random.default_rng(4).uniform(-1.3, 1.3, (most + 1000, dim)).astype(np.float32)
    p = C.params(method=C.STOCHASTIC, kernel=kernel, samples_per_subdomain=1, seed=9)

    def run(n):
        if grad:
            v, g, _, c = gpu.eval_grad(q[:n], p, contribs=True)
            return v, np.ascontiguousarray(g.T), c
        v, _, c = gpu.eval(q[:n], p, contribs=True)
        return v, v, c

    # 32 a warp (the last of 8 queries), 32 (13), 16 (all full), 16 (11), 16 (1), 8 (3)
    sizes = [most + 1000, most + 77, most, most - 5, most - 15, 128 * 8 * sms - 5]
    v, g, c = run(sizes[0])
    for n in sizes[1:]:
        a, b, d = run(n)
        assert bits_equal(a, v[:n]) and bits_equal(b, np.ascontiguousarray(g[..., :n]))
        assert np.array_equal(d, c[:n])
