"""Requests whose steps end inside a chunk, on its edge, across several and
across more than a warp's 32 at once: every checksum is the one of the
request's elements, in synchronous, pipelined and per-request ticks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 63, 64, 65, 255, 256, 257, 511, 512, 513, 2047, 2048, 2049, 8191, 8192, 8193, 16384, 20000]


@pytest.mark.parametrize("step", [1, 64, 100, 256, 257, 1000, 9000])
@pytest.mark.parametrize("form", ["sync", "pipelined", "each"])
def test_checksums_over_step_lengths(step, form):
    from mallocmc_gb300 import Allocator
    from mallocmc_gb300.policies import AlignmentPolicies, CreationPolicies, DistributionPolicies
    from mallocmc_gb300.serve import Server, expected_checksum

    lengths = np.array([n for n in LENGTHS if n <= 600 * step], dtype=np.int64)
    seeds = np.arange(11, 11 + len(lengths), dtype=np.int64)
    with Allocator(CreationPolicies.Scatter(pagesize=65536, accessblocksize=128 << 20),
                   DistributionPolicies.XMallocSIMD(65536), None, None, AlignmentPolicies.Shrink(16),
                   size=300 << 20) as alloc:
        srv = Server(alloc, slots=37, max_chunks=128, step=step, queue_cap=64)
        before = alloc.getAvailableSlots(16384)
        r = srv.run(np.zeros(len(lengths)), lengths, seeds, batched=form != "each", realtime=False,
                    pipelined=form == "pipelined")
        srv.close()
        assert r["completed"] == len(lengths)
        want = [expected_checksum(int(s), int(n)) for s, n in zip(seeds, lengths)]
        assert r["checksum"].tolist() == want
        assert alloc.getAvailableSlots(16384) == before and alloc.error_flags() == 0
