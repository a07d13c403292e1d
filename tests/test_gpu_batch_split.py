"""Batched brute force: a request's result is the same bits whether its tiles are summed
whole (large batches) or split into parts (small ones), at the edges of the parts."""
import numpy as np
import pytest

import sbh_capi as C
import sbh_workloads as W
from helpers import bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nq", [(16384, 3), (16385, 8), (16384 * 3 + 31, 17), (200003, 9),
                                  (2200000, 2)])
@pytest.mark.parametrize("dim,kernel", [(3, C.PLUMMER), (2, C.SMOOTH_DIST), (3, C.WINDING_NUMBER)])
def test_split_and_whole_tiles_agree(n, nq, dim, kernel):
    torch = pytest.importorskip("torch")
    pts, nrm, m = W.gaussian_mixture(n, seed=3, dim=dim)
    lo, hi = W.padded_box(pts)
    tree = C.GpuTree.build(pts, nrm, m, lo, hi, alpha=4.0)
    spts, snrm, sm = W.gaussian_mixture(5000, seed=4, dim=dim)
    slo, shi = W.padded_box(spts)
    small = C.GpuTree.build(spts, snrm, sm, slo, shi, alpha=4.0)
    p = C.params(method=C.BRUTE_FORCE, kernel=kernel)
    q = torch.from_numpy(np.ascontiguousarray(W.uniform_queries(nq, seed=5, dim=dim).T)).cuda()
    mass = torch.linspace(0.5, 1.0, nq, device="cuda")
    st = torch.cuda.current_stream().cuda_stream

    def run(extra):
        # `extra` queries on the small tree raise a warp's share of the batch
        out, cnt = torch.empty(nq, device="cuda"), torch.empty(nq, dtype=torch.int32, device="cuda")
        ent = [(tree, p, q.data_ptr(), nq, out.data_ptr(), cnt.data_ptr(), mass.data_ptr())]
        keep = []
        if extra:
            eq = torch.rand(dim, extra, device="cuda")
            eo = torch.empty(extra, device="cuda")
            keep = [eq, eo]
            ent.append((small, p, eq.data_ptr(), extra, eo.data_ptr(), 0, 0))
        C.eval_batch(ent, stream=st)
        torch.cuda.synchronize()
        assert (cnt == n).all()
        return out.cpu().numpy()

    alone = run(0)
    whole = run(2000000 if n > 10 ** 6 else 400000)  # shares of over 8 n sources
    assert bits_equal(alone, whole)
    assert bits_equal(alone, run(0))  # counters are back at zero
    want = tree.eval(W.uniform_queries(nq, seed=5, dim=dim), p)[0].astype(np.float64)
    # own terms (a source of the given mass at the query point), as the batch subtracts them
    self_value = {C.PLUMMER: mass.cpu().numpy() / 1e-3, C.SMOOTH_DIST: np.ones(nq),
                  C.WINDING_NUMBER: np.zeros(nq)}[kernel].astype(np.float64)
    scale = np.abs(want) + self_value + (1.0 if kernel == C.WINDING_NUMBER else 0.0)
    assert (np.abs(alone - (want - self_value)) <= 2e-6 * scale).all()
