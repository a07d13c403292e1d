"""Batches of changing make-up (each its own graph) while other threads build and destroy
trees, which synchronises the device."""
import threading

import numpy as np
import pytest

import sbh_capi as C
import sbh_workloads as W

pytestmark = pytest.mark.gpu


def test_batches_beside_tree_builds():
    torch = pytest.importorskip("torch")
    pts, nrm, m = W.gaussian_mixture(4000, seed=1)
    lo, hi = W.padded_box(pts)
    tree = C.GpuTree.build(pts, nrm, m, lo, hi, alpha=3.0, dim_split_log=2)
    server = C.Server(slots=2, slot_queries=4096)
    tid = server.add_tree(tree)
    stop, bad = threading.Event(), []

    def churn():
        try:
            while not stop.is_set():
                C.GpuTree.build(pts, nrm, m, lo, hi).close()
        except Exception as e:  # noqa: BLE001
            bad.append(e)

    threads = [threading.Thread(target=churn) for _ in range(2)]
    [t.start() for t in threads]
    try:
        rng = np.random.default_rng(2)
        q = rng.uniform(-1, 1, (700, 3)).astype(np.float32)
        kinds = [(C.BARNES_HUT, k) for k in range(4)] + [(C.BRUTE_FORCE, k) for k in range(4)] + [
            (C.STOCHASTIC, 0)]
        for mask in range(1, 1 << 9, 7):
            reqs = [(server.submit(tid, q, C.params(method=a, kernel=k)), a, k)
                    for i, (a, k) in enumerate(kinds) if mask >> i & 1]
            for r, a, k in reqs:
                assert np.isfinite(r.wait()).all()
    finally:
        stop.set()
        [t.join() for t in threads]
    assert not bad
    server.close()
