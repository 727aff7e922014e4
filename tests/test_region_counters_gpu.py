"""A multi-page free resets the counters of the regions its pages lie in: after
chunk walks have found a full heap and raised every region's counter, chunks
are served again from the freed run's pages, wherever in the heap they are."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pages", [2, 15, 16, 17, 40])
def test_multi_page_free_opens_its_regions(pages):
    from mallocmc_gb300 import Allocator
    from mallocmc_gb300.policies import CreationPolicies
    from mallocmc_gb300.workloads import alloc_offsets, free_offsets

    with Allocator(CreationPolicies.Scatter(accessblocksize=8 << 20), size=32 << 20) as alloc:
        total = alloc.geometry().numpages
        size = np.array([pages * 4096], dtype=np.uint32)
        runs = [alloc_offsets(alloc, 1, 1, size, i) for i in range(4)]
        first = [int(o.cpu().item()) // 4096 for _, o in runs]
        assert min(first) >= 0
        # every other page formatted for 2048-byte chunks, and more requests than fit
        n = 2 * (total - 4 * pages) + 64
        _, offs = alloc_offsets(alloc, -(-n // 32), 32, np.full(-(-n // 32) * 32, 2048, dtype=np.uint32), 9)
        assert int((offs >= 0).sum().item()) == 2 * (total - 4 * pages)
        regions = alloc.snapshot()[1]
        lo, hi = first[2] // 16, (first[2] + pages - 1) // 16
        # a failing walk raises every region it leaves (of several at once, one does)
        assert np.all(regions[lo: hi + 1] >= 1)
        assert free_offsets(alloc, 1, 1, *runs[2], 2) == 0
        ptes, regions, _, _ = alloc.snapshot()
        assert np.all(regions[lo: hi + 1] == 0) and np.all(ptes[first[2]: first[2] + pages, 0] == 0)
        _, again = alloc_offsets(alloc, 1, 1, np.array([2048], dtype=np.uint32), 10)
        assert first[2] <= int(again.cpu().item()) // 4096 < first[2] + pages
        assert alloc.error_flags() == 0
