"""The stress's payload where its split can go wrong: block lengths around a
16-byte unit, a 32-byte pair, a 256-byte piece and the 1 KiB a pass covers,
lanes without a whole unit, and blocks longer than a pass. Every pair completes,
no word mismatches, and the checksum is the one that follows from the pattern
words (u64 arithmetic, computed here with numpy)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGES = [16, 32, 48, 240, 256, 272, 496, 512, 528, 1008, 1024, 1040, 2032, 2048, 2064, 3072]


def expected_checksum(sizes, seed, warp):
    """sizes[round, thread]: XOR over the threads of each one's sum, over its
    rounds, of (m + 2i) ^ (m + 2i + 1) per unit i of its block; for the warp
    pattern unit i counts for the warp's lane i % 32."""
    from mallocmc_gb300.seeds import mix64

    rounds, threads = sizes.shape
    sums = np.zeros(threads, dtype=np.uint64)
    with np.errstate(over="ignore"):
        for r in range(rounds):
            m = mix64(seed, np.arange(threads, dtype=np.uint64), r)
            for t in range(threads):
                i = np.arange(sizes[r, t] // 16, dtype=np.uint64)
                x = m[t] + np.uint64(2) * i
                c = x ^ (x + np.uint64(1))
                if warp:
                    np.add.at(sums, (t & ~31) + (i % np.uint64(32)).astype(np.int64), c)
                else:
                    sums[t] += c.sum(dtype=np.uint64)
    return int(np.bitwise_xor.reduce(sums))


@pytest.mark.parametrize("warp", [False, True])
@pytest.mark.parametrize("draw", ["edges", "one", "units"])
def test_checksum_of_block_lengths(warp, draw):
    from mallocmc_gb300 import Allocator
    from mallocmc_gb300.policies import CreationPolicies
    from mallocmc_gb300.workloads import PATTERN_THREAD, PATTERN_WARP, run_stress

    rng = np.random.default_rng(11)
    blocks, tpb, rounds, seed = 3, 96, 4, 17
    shape = (rounds, blocks * tpb)
    sizes = {"edges": rng.choice(EDGES, size=shape), "one": np.full(shape, 3072),
             "units": rng.integers(1, 400, size=shape)}[draw].astype(np.uint16)
    with Allocator(CreationPolicies.Scatter(accessblocksize=32 << 20), size=128 << 20) as alloc:
        r = run_stress(alloc, blocks, tpb, rounds, seed=seed, sizes=sizes,
                       write_pattern=PATTERN_WARP if warp else PATTERN_THREAD)
    assert r["pairs"] == sizes.size and r["nulls"] == 0 and r["bad"] == 0
    assert r["checksum"] == expected_checksum(sizes.astype(np.int64), seed, warp)
