"""Chunk walks past multi-page runs: they pass the regions that runs fill by a
bitmap of the pages outside runs, and full regions several at a time. Whatever
the region size (with 12, no bitmap word holds a region and the bitmap is not
used) and whichever path placed and freed the runs, every page outside a live
run is found, and none inside one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PAGE = 4096


@pytest.mark.parametrize("tpb", [32, 24])  # whole warps: served together; partial ones: lock-free
@pytest.mark.parametrize("regionsize", [4, 8, 12, 16, 32])
def test_chunks_find_every_page_outside_runs(regionsize, tpb):
    import torch

    from mallocmc_gb300 import Allocator
    from mallocmc_gb300.policies import CreationPolicies
    from mallocmc_gb300.workloads import alloc_offsets, free_offsets

    with Allocator(CreationPolicies.Scatter(accessblocksize=8 << 20, regionsize=regionsize, reference_quirks=False),
                   size=64 << 20) as alloc:
        rng = np.random.default_rng(regionsize + tpb)
        total = alloc.geometry().numpages
        blocks = -(-total // (21 * tpb))
        sizes = (rng.integers(2, 40, blocks * tpb) * PAGE).astype(np.uint32)
        ds, offs = alloc_offsets(alloc, blocks, tpb, sizes, 1)
        for seed in (2, 3):  # among the runs; and among what is left of them after frees
            at = offs.cpu().numpy()
            used = np.zeros(total, dtype=bool)
            for a, s in zip(at[at >= 0] // PAGE, sizes[at >= 0] // PAGE):
                assert not used[a : a + s].any()
                used[a : a + s] = True
            free = int((~used).sum())
            chunks = np.full(32 * max(1, -(-2 * free // 32)), 2048, dtype=np.uint32)  # (the runs may leave no page)
            chunks[2 * free :] = 0
            cds, coffs = alloc_offsets(alloc, len(chunks) // 32, 32, chunks, seed)
            got = coffs.cpu().numpy()[: 2 * free]
            single = []
            for _ in range(2 * free - int((got >= 0).sum())):  # passed over while another's claim was in the way
                single.append(alloc_offsets(alloc, 1, 1, np.array([2048], dtype=np.uint32), 9))
            every = np.concatenate([got[got >= 0]] + [o.cpu().numpy() for _, o in single])
            assert len(np.unique(every)) == 2 * free and (every >= 0).all()
            assert not used[every // PAGE].any()
            _, none = alloc_offsets(alloc, 1, 1, np.array([2048], dtype=np.uint32), 9)
            assert int(none.cpu().item()) == -1
            assert free_offsets(alloc, len(chunks) // 32, 32, cds, coffs, seed) == 0
            for d, o in single:
                assert free_offsets(alloc, 1, 1, d, o, 9) == 0
            victims = torch.from_numpy((rng.random(len(at)) < 0.4) & (at >= 0)).cuda()
            assert free_offsets(alloc, blocks, tpb, ds, torch.where(victims, offs, torch.full_like(offs, -1)), 1) == 0
            offs = torch.where(victims, torch.full_like(offs, -1), offs)
        assert alloc.error_flags() == 0
