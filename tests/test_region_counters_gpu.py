"""The region counters under concurrent ids: a walk that finds nothing counts in
regions with no page and no chunk free, and leaves those alone that have room
for another size; the heap's second pass counts nowhere."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("regionsize", [8, 16, 32])
def test_failed_walks_count_in_full_regions_only(regionsize):
    from mallocmc_gb300 import Allocator
    from mallocmc_gb300.policies import CreationPolicies
    from mallocmc_gb300.workloads import alloc_offsets, free_offsets

    with Allocator(CreationPolicies.Scatter(accessblocksize=8 << 20, regionsize=regionsize),
                   size=32 << 20) as alloc:
        total = alloc.geometry().numpages
        n = 2 * total
        ds, offs = alloc_offsets(alloc, n // 32, 32, np.full(n, 2048, dtype=np.uint32), 1)
        pages = offs.cpu().numpy() // 4096
        assert pages.min() >= 0  # two chunks on every page
        # one chunk back on every 200th page
        victims = np.isin(pages, np.arange(0, total, 200)) & (offs.cpu().numpy() % 4096 == 0)
        import torch

        part = torch.where(torch.from_numpy(victims).cuda(), offs, torch.full_like(offs, -1))
        assert free_offsets(alloc, n // 32, 32, ds, part, 1) == 0
        before = alloc.snapshot()[1].astype(np.int64)
        for seed in range(3):  # a whole page: no region has one, many have room for less
            _, got = alloc_offsets(alloc, 1, 1, np.array([4096], dtype=np.uint32), seed)
            assert int(got.cpu().item()) == -1
        after = alloc.snapshot()[1].astype(np.int64)
        room = np.zeros(len(before), dtype=bool)
        room[np.arange(0, total, 200) // regionsize] = True
        assert np.array_equal(after[room], before[room])
        level = 3 * regionsize // 4
        assert np.array_equal(after[~room], np.where(before[~room] < level, np.minimum(before[~room] + 3, level),
                                                     before[~room]))
        _, again = alloc_offsets(alloc, 1, 1, np.array([2048], dtype=np.uint32), 5)
        assert int(again.cpu().item()) // 4096 % 200 == 0
        assert alloc.error_flags() == 0
