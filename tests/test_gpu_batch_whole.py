"""Batched brute force in batches so large that a request's tiles are summed whole: the same bits
as where each part of a tile is a work unit of its own."""
import numpy as np
import pytest

import sbh_capi as C
import sbh_workloads as W
from helpers import bits_equal

pytestmark = pytest.mark.gpu
TILE = 8  # queries


@pytest.mark.parametrize("n,dim,kernel", [
    (16385, 3, C.GRAVITY), (16385, 2, C.WINDING_NUMBER), (16384 * 3 + 31, 2, C.SMOOTH_DIST),
    (16384 * 3 + 31, 3, C.WINDING_NUMBER), (200003, 3, C.PLUMMER), (2200000, 3, C.PLUMMER)])
def test_whole_tiles_equal_split_ones(n, dim, kernel):
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    pts, nrm, m = W.gaussian_mixture(n, seed=3, dim=dim)
    lo, hi = W.padded_box(pts)
    tree = C.GpuTree.build(pts, nrm, m, lo, hi, alpha=4.0)
    p = C.params(method=C.BRUTE_FORCE, kernel=kernel)
    nq = 77
    q = torch.from_numpy(np.ascontiguousarray(W.uniform_queries(nq, seed=5, dim=dim).T)).cuda()
    mass = torch.linspace(0.5, 1.0, nq, device="cuda")
    # A tile is split where its sources exceed an eighth of a warp's share of the batch, and an
    # SM has 64 warps at most: never with `extra` more queries on the same tree, and always
    # with the request alone, whose 10 tiles leave each of the 16 warps or more of an SM less
    # than 10 n / 16 / SMs sources.
    extra = 8 * TILE * 64 * sms + TILE + 5
    assert 10 / (16 * sms) < 8 <= extra / TILE / (64 * sms)

    def run(queries, mass, more=None):
        k = queries.shape[1]
        out = torch.full((k,), float("nan"), device="cuda")
        cnt = torch.zeros(k, dtype=torch.int32, device="cuda")
        ptr = mass.data_ptr() if mass is not None else 0
        batch = [(tree, p, queries.data_ptr(), k, out.data_ptr(), cnt.data_ptr(), ptr)]
        values = None
        if more is not None:
            values = torch.full((more.shape[1],), float("nan"), device="cuda")
            batch.append((tree, p, more.data_ptr(), more.shape[1], values.data_ptr(), 0, 0))
        torch.cuda.synchronize()
        C.eval_batch(batch, stream=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert (cnt == n).all()
        return out.cpu().numpy(), values

    split, _ = run(q, mass)
    more = torch.rand(dim, extra, device="cuda")
    whole, values = run(q, mass, more)
    assert bits_equal(whole, split)
    # and the last tiles of the large request, the ragged one among them, split
    tail, _ = run(more[:, -75:].contiguous(), None)
    assert bits_equal(values[-75:].cpu().numpy(), tail)
