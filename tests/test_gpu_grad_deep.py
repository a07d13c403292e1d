"""Barnes-Hut gradients on trees as deep as they may be (duplicate points reach any depth cap):
a lane per query and the warp vote, on both sides of the shared-memory size that needs no opt-in."""
import numpy as np
import pytest

import oracle as O
import sbh_capi as C
import sbh_workloads as W
from helpers import bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("depth", [766, 767, 1000])
@pytest.mark.parametrize("kernel", [C.GRAVITY, C.PLUMMER])
@pytest.mark.parametrize("method", ["vote", "lane"])
def test_deep_trees(depth, kernel, method):
    torch = pytest.importorskip("torch")
    pts, nrm, m = W.gaussian_mixture(300, seed=2)
    pts[1] = pts[0]
    lo, hi = W.padded_box(pts)
    gpu = C.GpuTree(C.HostTree(pts, nrm, m, lo, hi, max_depth=depth))
    assert gpu.info.depth == depth
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    nq = 70 if method == "vote" else 2048 * sms + 1  # beyond a warp per query
    meth = C.BARNES_HUT_VOTE if method == "vote" else C.BARNES_HUT
    q = W.uniform_queries(nq, seed=3)
    # every leaf is opened: the values are the plain walk's bits, the gradients the exact sum's
    p = C.params(method=meth, kernel=kernel, beta=float("inf"))
    v, g, _, c = gpu.eval_grad(q, p, contribs=True)
    pv, _, pc = gpu.eval(q, p, contribs=True)
    assert bits_equal(v, pv) and np.array_equal(c, pc)
    ov, og = O.brute_force_grad_f64(pts, m, kernel, q[:300])
    assert np.all(np.abs(v[:300] - ov) <= 1e-5 * np.abs(ov))
    err = np.linalg.norm(g[:300].astype(np.float64) - og, axis=1)
    assert np.all(err <= 1e-4 * np.linalg.norm(og, axis=1) + 1e-30)
