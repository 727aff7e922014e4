"""Regions whose counters pass a byte's range (3/4 of 342 pages is 256): failed
walks of one device thread with the reference's serial ids count and pass them as
the oracle does, up to their limit and beyond; then frees and new requests."""
import numpy as np
import pytest

from oracle.oracle import HeapConfig, OracleHeap
from tests.test_parity_gpu import gpu_allocator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("regionsize", [340, 342, 400, 512])
@pytest.mark.parametrize("fails", [120, 160, 230, 330])
def test_counters_of_large_regions(regionsize, fails):
    from mallocmc_gb300.workloads import run_program

    cfg = HeapConfig(1024, 2 * regionsize * 1024, regionsize, 2, False)
    heap = 3 * (regionsize * (12 + 1024) + 4) + 4096
    oh = OracleHeap(cfg, heap)
    pages = oh.numpages
    ops = [("m", 1000)] * (pages + fails)
    ops += [("f", i) for i in (0, pages // 2, pages - 1)] + [("m", 900)] * 3 + [("m", 1000)] * 3
    offs, want = [], []
    for k, a in ops:
        if k == "m":
            offs.append(oh.malloc(a))
            want.append(offs[-1])
        else:
            oh.free_offset(offs[a])
            want.append(0)
    assert sum(o < 0 for o in offs) == fails + 3
    with gpu_allocator(cfg, heap) as alloc:
        out = run_program(alloc, ops)
        snap = alloc.snapshot()
    assert np.array_equal(out, np.array(want, dtype=np.int64))
    ptes, regions, masks = oh.snapshot()
    assert np.array_equal(snap[0], ptes)
    assert np.array_equal(snap[1], regions)
    assert np.array_equal(snap[2], masks)
    assert snap[3] == oh.header()
