"""The slot scan's loads and run words at their edges: heaps whose page count is
not a multiple of 4, 32 or 1024 pages, region sizes that are odd, states with
runs across words, tiles and blocks of the scan; the count of every size equals
the oracle's on the same state."""
import numpy as np
import pytest

from oracle.oracle import HeapConfig, OracleHeap
from tests.test_parity_gpu import gpu_allocator

pytestmark = pytest.mark.gpu

SIZES = [1, 16, 100, 129, 500, 1024, 2048, 3000, 4095, 4096, 4097, 8192, 3 * 4096, 7 * 4096, 29 * 4096, 30 * 4096,
         31 * 4096, 33 * 4096, 64 * 4096, 100 * 4096, 1000 * 4096]


@pytest.mark.parametrize("regionsize, mib", [(1, 9), (3, 21), (7, 16), (16, 13), (32, 64), (16, 100)])
def test_counts_equal_the_oracles(regionsize, mib):
    from mallocmc_gb300.workloads import program_arrays, run_program

    cfg = HeapConfig(4096, 8 << 20, regionsize, 2, False)
    rng = np.random.default_rng(regionsize * 1000 + mib)
    with gpu_allocator(cfg, mib << 20) as alloc:
        oh = OracleHeap(cfg, mib << 20)
        assert [alloc.getAvailableSlots(s) for s in SIZES] == \
            oh.run_program(*[x if i else x.tobytes() for i, x in enumerate(program_arrays([("s", s) for s in SIZES]))]).tolist()
        n = 260
        sizes = np.where(rng.random(n) < 0.5, rng.integers(1, 4096, size=n), rng.integers(4097, 40 * 4096, size=n))
        ops = [("m", int(s)) for s in sizes] + [("f", int(i)) for i in rng.permutation(n)[: n // 2]]
        ops += [("s", s) for s in SIZES]
        kinds, args = program_arrays(ops)
        want = oh.run_program(kinds.tobytes(), args)
        got = run_program(alloc, ops)
        assert got[-len(SIZES):].tolist() == want[-len(SIZES):].tolist()
        assert [alloc.getAvailableSlots(s) for s in SIZES] == want[-len(SIZES):].tolist()
        oh.close()
