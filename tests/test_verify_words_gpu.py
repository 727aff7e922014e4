"""The verify workload's words at the edges of its 32-byte accesses: blocks of
0 to 24 words and a few longer ones, at every 16-byte offset in a sector. All
words read back; with another seed every word differs, and the count is exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("words", [range(0, 25), [31, 32, 33, 63, 64, 65, 150], [255, 256, 257, 1000]])
@pytest.mark.parametrize("coalesce", [True, False])
def test_words_written_read_and_counted(words, coalesce):
    from mallocmc_gb300 import Allocator
    from mallocmc_gb300.policies import CreationPolicies, DistributionPolicies
    from mallocmc_gb300.workloads import alloc_offsets, free_offsets

    sizes = 4 * np.random.default_rng(5).choice(list(words), size=640).astype(np.uint32)
    dist = DistributionPolicies.XMallocSIMD(4096) if coalesce else DistributionPolicies.Noop()
    with Allocator(CreationPolicies.Scatter(accessblocksize=16 << 20), dist, size=64 << 20) as alloc:
        for seed, other in ((3, 3), (3, 0x40000003)):
            ds, offs = alloc_offsets(alloc, 5, 128, sizes, seed)
            got = offs.cpu().numpy()
            assert np.all(got[sizes > 0] >= 0) and len(np.unique(got[sizes > 0] % 32)) == 2
            wrong = free_offsets(alloc, 5, 128, ds, offs, other)
            assert wrong == (0 if other == seed else int(sizes.sum()) // 4)
        assert alloc.error_flags() == 0
