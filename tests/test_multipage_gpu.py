"""Multi-page requests of whole warps, which one warp serves for all that wait:
runs of one length pack the heap without a page between them, whatever the
length's place among the words and windows of the bitmap search; mixed lengths
and chunks in one warp are disjoint and keep their patterns; everything freed
leaves the page table and its bitmap empty. Partial warps and requests beyond
the service's limit take the lock-free search on the same heap."""
import numpy as np
import pytest

from tests.test_verify_gpu import assert_all_free

pytestmark = pytest.mark.gpu

PAGE = 4096


def _heap(mib=64):
    from mallocmc_gb300 import Allocator
    from mallocmc_gb300.policies import CreationPolicies

    # the reference's hint wraps for good once a run starts at page 0: these heaps are filled down to it
    return Allocator(CreationPolicies.Scatter(accessblocksize=8 << 20, reference_quirks=False), size=mib << 20)


def _alloc(alloc, sizes, tpb, seed):
    from mallocmc_gb300.workloads import alloc_offsets

    n = -(-len(sizes) // tpb) * tpb
    padded = np.concatenate([sizes, np.zeros(n - len(sizes), dtype=np.uint32)]).astype(np.uint32)
    ds, offs = alloc_offsets(alloc, n // tpb, tpb, padded, seed)
    return ds, offs, padded, seed


def _free(alloc, got, tpb):
    from mallocmc_gb300.workloads import free_offsets

    ds, offs, padded, seed = got
    assert free_offsets(alloc, len(padded) // tpb, tpb, ds, offs, seed) == 0


def _assert_disjoint(offs, sizes):
    ok = offs >= 0
    order = np.argsort(offs[ok])
    lo, hi = offs[ok][order], (offs[ok] + (sizes[ok] + 15) // 16 * 16)[order]
    assert np.all(lo[1:] >= hi[:-1])


def _assert_empty(alloc):
    snap = alloc.snapshot()
    assert_all_free(snap)
    assert int(np.count_nonzero(snap[0][:, 0] > PAGE)) == 0
    assert np.all(alloc.freemap()[snap[0][:, 0] == 0])
    assert alloc.error_flags() == 0


@pytest.mark.parametrize("pages", [2, 3, 31, 32, 33, 64, 100, 1023, 1024])
def test_runs_of_one_length_pack_the_heap(pages):
    with _heap() as alloc:
        total = alloc.geometry().numpages
        want = total // pages
        sizes = np.full(want + 40, pages * PAGE, dtype=np.uint32)
        for seed in (1, 2):  # a fresh heap, and the one it leaves
            got = _alloc(alloc, sizes, 32, seed)
            offs = got[1].cpu().numpy()[: len(sizes)]
            assert int((offs >= 0).sum()) == want
            _assert_disjoint(offs, sizes)
            assert np.all(offs[offs >= 0] % PAGE == 0)
            _free(alloc, got, 32)
            _assert_empty(alloc)


@pytest.mark.parametrize("tpb", [32, 96, 128])
@pytest.mark.parametrize("most", [4, 60, 700])
def test_mixed_lengths_and_chunks(most, tpb):
    rng = np.random.default_rng(most + tpb)
    with _heap(256) as alloc:
        live = []
        for seed in range(6):
            n = min(1500, 40000 // most)
            sizes = np.where(rng.random(n) < 0.4, rng.integers(PAGE + 1, most * PAGE, size=n),
                             rng.integers(4, PAGE, size=n)).astype(np.uint32) // 4 * 4
            live.append(_alloc(alloc, sizes, tpb, seed))
            offs = np.concatenate([g[1].cpu().numpy() for g in live])
            _assert_disjoint(offs, np.concatenate([g[2] for g in live]).astype(np.int64))
            if seed in (2, 4):
                _free(alloc, live.pop(seed // 4), tpb)
        assert all(int((g[1].cpu().numpy()[g[2] > 0] >= 0).sum()) > 0 for g in live)
        for g in live:
            _free(alloc, g, tpb)
        _assert_empty(alloc)


@pytest.mark.parametrize("pages, tpb", [(1025, 32), (1200, 64), (5, 20), (40, 48)])
def test_lock_free_search_beside_the_service(pages, tpb):
    """Requests above the service's limit, or from warps with idle lanes (a
    block of 20, or of 48, threads), in one launch with whole warps' requests."""
    with _heap(256) as alloc:
        n = 4 * tpb
        sizes = np.full(n, 3 * PAGE, dtype=np.uint32)
        sizes[::5] = pages * PAGE
        sizes[::7] = 64
        got = _alloc(alloc, sizes, tpb, 3)
        offs = got[1].cpu().numpy()
        _assert_disjoint(offs, got[2].astype(np.int64))
        assert int((offs >= 0).sum()) >= n // 2
        _free(alloc, got, tpb)
        _assert_empty(alloc)


def test_more_requests_than_the_ring_holds():
    """Every thread of 77 824 asks at once, more than twice the ring's tickets;
    a second and third kernel run the ring around."""
    with _heap(1024) as alloc:
        total = alloc.geometry().numpages
        for seed in (1, 2, 3):
            got = _alloc(alloc, np.full(304 * 256, 3 * PAGE, dtype=np.uint32), 256, seed)
            offs = got[1].cpu().numpy()
            assert int((offs >= 0).sum()) == min(304 * 256, total // 3)
            _assert_disjoint(offs, got[2].astype(np.int64))
            _free(alloc, got, 256)
            _assert_empty(alloc)
