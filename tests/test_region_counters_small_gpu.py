"""Regions full of small chunks, whose on-page masks cost the page a chunk or two
of what its size divided by theirs would be: walks that find nothing count them
as full, up to the level from which later walks pass them. One chunk freed is
found again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _capacity(pagesize, size):
    """Chunks on a page with on-page masks: segments of 32 and a mask word each,
    and a last, shorter one (at most 31 chunks and its word)."""
    segment = 32 * size + 4
    full = min(32, pagesize // segment)
    rest = pagesize - full * segment - 4
    return 32 * full + (min(31, rest // size) if full != 32 and rest > 0 else 0)


@pytest.mark.parametrize("pagesize, size", [(4096, 16), (4096, 32), (4096, 48), (4096, 64), (65536, 256),
                                            (65536, 1024)])
def test_regions_full_of_small_chunks_count(pagesize, size):
    from mallocmc_gb300 import Allocator
    from mallocmc_gb300.policies import CreationPolicies, DistributionPolicies
    from mallocmc_gb300.workloads import alloc_offsets, free_offsets

    with Allocator(CreationPolicies.Scatter(pagesize=pagesize, accessblocksize=8 << 20),
                   DistributionPolicies.Noop(), size=17 << 20) as alloc:
        geo = alloc.geometry()
        total = geo.numpages * _capacity(pagesize, size)
        n = (total // 32 + 1) * 32
        sizes = np.full(n, size, dtype=np.uint32)
        ds, offs = alloc_offsets(alloc, n // 32, 32, sizes, 1)
        got = offs.cpu().numpy()
        held = int((got >= 0).sum())
        assert total - total // 100 <= held <= total
        while held < total:  # what concurrent walks passed
            _, more = alloc_offsets(alloc, 1, 1, sizes[:1], 1)
            assert int(more.cpu().item()) >= 0
            held += 1
        ptes, regions = alloc.snapshot()[:2]
        assert np.all(ptes[:, 0] == size) and np.all(ptes[:, 1] == _capacity(pagesize, size))
        level = 3 * alloc.creation.regionsize // 4
        for seed in range(level):
            _, none = alloc_offsets(alloc, 1, 1, sizes[:1], seed)
            assert int(none.cpu().item()) == -1
        assert np.all(alloc.snapshot()[1] == level)
        # one chunk back: the second pass finds it in a region the first one passes
        import torch

        one = torch.where(torch.arange(n, device=offs.device) == int(np.argmax(got >= 0)), offs,
                          torch.full_like(offs, -1))
        assert free_offsets(alloc, n // 32, 32, ds, one, 1) == 0
        _, again = alloc_offsets(alloc, 1, 1, sizes[:1], 3)
        assert int(again.cpu().item()) == int(got[np.argmax(got >= 0)])
        assert alloc.error_flags() == 0
