"""Device memory for the build's workspace or for the tree, but not for both: the build takes place on
the host, whose tree needs its own memory alone."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

# In a process of its own: the library's pool starts empty, and the card is filled but for `room`.
CHILD = """
import numpy as np, torch
import sbh_capi as C, sbh_workloads as W
n = 1 << 22
pts, nrm, m = W.torus_surface(n, 1)
lo, hi = W.padded_box(pts)
want = C.GpuTree(C.HostTree(pts, nrm, m, lo, hi))
q, p = W.uniform_queries(500, seed=1), C.params(method=C.BARNES_HUT, kernel=C.WINDING_NUMBER)
value = want.eval(q, p)[0]
info = want.info  # the tree stays: closed, its memory would be the pool's to give
small = C.GpuTree.build(pts[:1000], nrm[:1000], m[:1000], lo, hi)
small.eval(q, p)
# the workspace: about 254 bytes a point (70 for points, 92 for each of 2 n nodes)
room = 254 * n + info.device_bytes // 2
filler = []
while torch.cuda.mem_get_info()[0] > room + (64 << 20):
    filler.append(torch.empty(torch.cuda.mem_get_info()[0] - room - (32 << 20), dtype=torch.uint8,
                              device="cuda"))
got = C.GpuTree.build(pts, nrm, m, lo, hi)
assert not got.built_on_device
assert (got.info.num_nodes, got.info.depth) == (info.num_nodes, info.depth)
assert np.array_equal(got.eval(q, p)[0], value)
del filler, got, want
torch.cuda.empty_cache()
again = C.GpuTree.build(pts, nrm, m, lo, hi)
assert again.built_on_device and np.array_equal(again.eval(q, p)[0], value)
print("fallback ok")
"""


def test_tree_does_not_fit_beside_the_workspace():
    pytest.importorskip("torch")
    here = os.path.dirname(os.path.abspath(__file__))
    pkg = os.path.join(os.path.dirname(here), "stochastic-barnes-hut_b200")
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=here, capture_output=True, text=True,
                       timeout=300, env=dict(os.environ, PYTHONPATH=pkg))
    assert r.returncode == 0 and "fallback ok" in r.stdout, r.stdout + r.stderr
