"""Per-thread patterns of 16 to 256 bytes on grids of several waves, where the
lanes of a warp part and meet the most often: some requests join others, some
hash to a page of their own, some walk. Every launch ends with every pair made
and verified."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks", [1216, 2500, 4000])
@pytest.mark.parametrize("simd", [True, False])
def test_small_blocks_on_many_warps(blocks, simd):
    from mallocmc_gb300 import Allocator
    from mallocmc_gb300.policies import CreationPolicies, DistributionPolicies
    from mallocmc_gb300.workloads import PATTERN_THREAD, run_stress

    with Allocator(CreationPolicies.Scatter(accessblocksize=1 << 30),
                   None if simd else DistributionPolicies.Noop(), size=4 << 30) as alloc:
        for seed in range(6):
            st = run_stress(alloc, blocks, 256, 4, 16, 256, 16, seed=seed, write_pattern=PATTERN_THREAD)
            assert st["pairs"] == blocks * 256 * 4 and not st["nulls"] and not st["bad"]
        assert alloc.error_flags() == 0
