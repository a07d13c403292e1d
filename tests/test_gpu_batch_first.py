"""The first batch of a new engine while the default stream is busy: what the engine keeps
between its kernels is cleared on the stream that runs the batch, so a split brute-force request
gets its sums whatever is queued elsewhere."""
import numpy as np
import pytest

import sbh_capi as C
import sbh_workloads as W

pytestmark = pytest.mark.gpu
N = 200003  # 13 parts a tile


@pytest.fixture(scope="module")
def tree():
    pts, nrm, m = W.gaussian_mixture(N, seed=3)
    lo, hi = W.padded_box(pts)
    return C.GpuTree.build(pts, nrm, m, lo, hi, alpha=4.0)


def _busy(torch):
    """About a tenth of a second of work on the default stream (a bounded spin)."""
    torch.cuda._sleep(200_000_000)


# Sums of positive terms, each to a few FP32 roundings and compensated, by two schedules: 2e-6.
@pytest.mark.parametrize("kernel", [C.PLUMMER, C.SMOOTH_DIST])
def test_server(tree, kernel):
    torch = pytest.importorskip("torch")
    p = C.params(method=C.BRUTE_FORCE, kernel=kernel)
    q = W.uniform_queries(1001, seed=5)
    want, _ = tree.eval(q, p)
    for _ in range(3):
        server = C.Server(slots=1, slot_queries=4096)
        tid = server.add_tree(tree)
        _busy(torch)
        got = server.submit(tid, q, p).wait()
        assert np.all(np.abs(got - want) <= 2e-6 * np.abs(want))
        again = server.submit(tid, q, p).wait()
        assert np.array_equal(got, again)
        server.close()
        torch.cuda.synchronize()


def test_eval_batch(tree):
    """Growing requests make the device's engine anew; the caller's stream does not wait for the
    default one."""
    torch = pytest.importorskip("torch")
    p = C.params(method=C.BRUTE_FORCE, kernel=C.PLUMMER)
    stream = torch.cuda.Stream()
    for nq in (100, 70001, 150001):
        q = W.uniform_queries(nq, seed=nq)
        want, _ = tree.eval(q, p)
        d = torch.from_numpy(np.ascontiguousarray(q.T)).cuda()
        out = torch.empty(nq, device="cuda")
        torch.cuda.synchronize()
        _busy(torch)
        C.eval_batch([(tree, p, d.data_ptr(), nq, out.data_ptr(), 0, 0)], stream=stream.cuda_stream)
        stream.synchronize()
        with torch.cuda.stream(stream):
            got = out.cpu().numpy()
        assert np.all(np.abs(got - want) <= 2e-6 * np.abs(want))
        torch.cuda.synchronize()
