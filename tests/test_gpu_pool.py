"""The memory pool keeps what a build freed, for the next one, whatever trees are resident, and no
more than its 1 GiB of it."""
import pytest

import sbh_capi as C
import sbh_workloads as W

pytestmark = pytest.mark.gpu
MIB = 1 << 20
SLACK = 128 * MIB  # the driver's allocation granularity, and what else maps memory meanwhile


def test_freed_memory_is_kept_beside_resident_trees():
    torch = pytest.importorskip("torch")
    pts, nrm, m = W.torus_surface(1 << 20, 1)
    lo, hi = W.padded_box(pts)

    def build():
        return C.GpuTree.build(pts, nrm, m, lo, hi)

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    size = build().info.device_bytes
    assert size > SLACK  # a tree mapped afresh shows
    resident = [build() for _ in range(3 * 1024 * MIB // size + 1)]
    build().close()  # what it used is free in the pool
    before = free()
    tree = build()
    assert abs(free() - before) < SLACK  # served from there
    tree.close()
    assert abs(free() - before) < SLACK
    for t in resident:
        t.close()
    assert free() - before >= len(resident) * size - 1024 * MIB - SLACK
