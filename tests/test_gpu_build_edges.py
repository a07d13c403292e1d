"""The GPU tree build at its edges: levels on both sides of the shared-memory counting,
chains of single-child nodes that outgrow the first workspace, points outside the box."""
import threading

import numpy as np
import pytest

import sbh_capi as C
import sbh_workloads as W
from helpers import bits_equal

pytestmark = pytest.mark.gpu


def _same(pts, dim, dsl, lo, hi):
    rng = np.random.default_rng(2)
    nrm = rng.normal(size=pts.shape).astype(np.float32)
    m = rng.uniform(0.5, 1.5, len(pts)).astype(np.float32)
    ref = C.GpuTree(C.HostTree(pts, nrm, m, lo, hi, dim_split_log=dsl))
    got = C.GpuTree.build(pts, nrm, m, lo, hi, dim_split_log=dsl)
    # clamped points can share a leaf at the depth cap: the host's part of the contract
    assert got.built_on_device or ref.info.depth == 100
    for f in ("num_points", "num_nodes", "depth", "root_children"):
        assert getattr(got.info, f) == getattr(ref.info, f), f
    a, b = ref.export(), got.export()
    for k in a:
        assert bits_equal(a[k], b[k]), k


@pytest.mark.parametrize("dim,dsl", [(2, 1), (2, 3), (3, 1), (3, 2), (3, 3)])
@pytest.mark.parametrize("kind", ["chain", "outside", "grid", "large"])
def test_edges(dim, dsl, kind):
    rng = np.random.default_rng(7)
    if kind == "chain":  # pairs 2e-6 apart: up to ~20 levels of one child per pair
        a = rng.uniform(0.1, 1, (1500, dim))
        pts = np.concatenate([a, a + 2e-6]).astype(np.float32)
        pts = np.unique(pts, axis=0)
    elif kind == "outside":  # clamped to the outer cells
        pts = rng.normal(0, 1.0, (3000, dim)).astype(np.float32)
    elif kind == "grid":  # on cell borders
        k = np.arange(16) / 16.0
        pts = np.stack(np.meshgrid(*[k] * dim), -1).reshape(-1, dim).astype(np.float32)
    else:
        pts = rng.uniform(-1, 1, (150001, dim)).astype(np.float32)
    _same(pts, dim, dsl, np.full(dim, -1, np.float32), np.full(dim, 1, np.float32))


def test_builds_in_several_threads():
    pts, nrm, m = W.torus_surface(20000, seed=4)
    lo, hi = W.padded_box(pts)
    want = C.GpuTree(C.HostTree(pts, nrm, m, lo, hi, dim_split_log=2)).export()
    bad = []

    def work():
        for _ in range(3):
            got = C.GpuTree.build(pts, nrm, m, lo, hi, dim_split_log=2).export()
            if not all(bits_equal(want[k], got[k]) for k in want):
                bad.append(1)

    threads = [threading.Thread(target=work) for _ in range(6)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not bad
