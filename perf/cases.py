"""The work that users of the heap have it do, as measurable cases.

Six kinds, each through the package's public entry points (the Python mirror and
the C ABI under it):

  stress   a kernel whose threads each run rounds of malloc, write a pattern,
           read it back, free
  live     one kernel allocates a block per thread and fills it, a later kernel
           verifies and frees them: data that outlives its kernel
  frag     mixed small and multi-page requests: waves that fill part of the heap,
           a seeded half freed, another wave, every block's tags checked, all freed
  batch    many uneven jobs in one persistent launch, with their per-job results
  serve    a burst of requests through the continuous-batching loop
  slots    getAvailableSlots for several sizes on a partly used heap

Placements depend on which SM and warp a thread runs on, so the outputs are what
does not: counts, checksums, per-thread sizes, slot counts.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from mallocmc_gb300 import _lib as L
from mallocmc_gb300.allocator import Allocator
from mallocmc_gb300.autotune import GB300_FRAG_TUNED, GB300_TUNED, _accessblock, frag_allocator
from mallocmc_gb300.batch import Batch, expected_pairs, make_jobs
from mallocmc_gb300.fragmentation import frag_params, mean_request_bytes
from mallocmc_gb300.policies import AlignmentPolicies, CreationPolicies, DistributionPolicies
from mallocmc_gb300.serve import Server, expected_checksum, make_requests
from mallocmc_gb300.workloads import PATTERN_THREAD, PATTERN_WARP, launch_stress, run_program, stress_params

MIB = 1 << 20


def listed():
    return [
        # a small kernel on a small heap: the launch and one chain of round trips
        {"name": "stress_tiny", "kind": "stress", "heap_mib": 64, "accessblock_mib": 32, "blocks": 4, "threads": 64,
         "rounds": 2, "lo": 16, "hi": 1024, "step": 16, "warp": False, "table": False, "coalesce": True,
         "reset": False},
        # the benchmark: the whole GPU, sizes 16 to 1024 from a table
        {"name": "stress_uniform", "kind": "stress", "heap_mib": 8192, "accessblock_mib": 4096, "blocks": 1216,
         "threads": 256, "rounds": 100, "lo": 16, "hi": 1024, "step": 16, "warp": True, "table": True,
         "coalesce": True, "reset": False},
        # small objects of many sizes, joined per warp; a grid that fills no whole number of waves
        {"name": "stress_small_objects", "kind": "stress", "heap_mib": 4096, "accessblock_mib": 2048, "blocks": 701,
         "threads": 224, "rounds": 40, "lo": 16, "hi": 112, "step": 16, "warp": False, "table": False,
         "coalesce": True, "reset": False},
        # every thread allocates the same structure
        {"name": "stress_one_size", "kind": "stress", "heap_mib": 4096, "accessblock_mib": 2048, "blocks": 608,
         "threads": 256, "rounds": 40, "lo": 208, "hi": 208, "step": 16, "warp": True, "table": False,
         "coalesce": True, "reset": False},
        # the other policies: no distribution, pages given back when their last chunk goes
        {"name": "stress_noop_reset", "kind": "stress", "heap_mib": 2048, "accessblock_mib": 1024, "blocks": 333,
         "threads": 160, "rounds": 20, "lo": 16, "hi": 2000, "step": 8, "warp": False, "table": False,
         "coalesce": False, "reset": True},
        # nodes of a data structure that one kernel builds and a later one takes down
        {"name": "live_nodes", "kind": "live", "heap_mib": 4096, "accessblock_mib": 2048, "blocks": 3907,
         "threads": 256, "lo": 8, "hi": 600},
        # mixed request sizes on a heap that stays in use
        {"name": "frag_mixed", "kind": "frag", "heap_mib": 8192, "blocks": 304, "threads": 256, "waves": 3,
         "small_hi": 2048, "large_lo": 8192, "large_hi": 1 << 20, "large_permille": 100},
        {"name": "frag_small", "kind": "frag", "heap_mib": 512, "blocks": 12, "threads": 256, "waves": 3,
         "small_hi": 2048, "large_lo": 8192, "large_hi": 1 << 20, "large_permille": 100},
        # the uneven-job workload on the tuned geometry, and a small one on the reference's defaults
        {"name": "batch_512_jobs", "kind": "batch", "heap_mib": 16384, "tuned": True, "jobs": 512, "tmin": 32,
         "tmax": 65536, "mean_size": 64, "max_size": 4096, "max_cycles": 16},
        {"name": "batch_24_jobs", "kind": "batch", "heap_mib": 4096, "tuned": False, "jobs": 24, "tmin": 32,
         "tmax": 4096, "mean_size": 64, "max_size": 4096, "max_cycles": 16},
        # requests that all arrive at once, served by pipelined ticks
        {"name": "serve_burst", "kind": "serve", "heap_mib": 65536, "requests": 6000, "median": 1024,
         "pipelined": True},
        # a program that sizes its work by what the heap still holds
        {"name": "slots_queries", "kind": "slots", "heap_mib": 65536, "ops": 600},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["stress", "stress", "stress", "live", "frag", "batch", "serve", "slots"])
    if kind == "stress":
        threads = rng.choice([32, 64, 96, 128, 160, 224, 256])
        blocks = _log(rng, 2, 1216)
        lo = 16 * rng.randint(1, 16)
        hi = lo if rng.random() < 0.2 else 16 * rng.randint(lo // 16, 64)
        return {"kind": "stress", "heap_mib": rng.choice([4096, 6144, 8192]), "accessblock_mib": 2048,
                "blocks": blocks, "threads": threads, "rounds": _log(rng, 2, 80), "lo": lo, "hi": hi, "step": 16,
                "warp": rng.random() < 0.5, "table": rng.random() < 0.5, "coalesce": rng.random() < 0.8,
                "reset": rng.random() < 0.2}
    if kind == "live":
        return {"kind": "live", "heap_mib": 4096, "accessblock_mib": 2048, "blocks": _log(rng, 3, 3907),
                "threads": rng.choice([96, 128, 256]), "lo": 8 * rng.randint(1, 8), "hi": rng.randint(70, 600)}
    if kind == "frag":
        heap = rng.choice([512, 1024, 2048, 4096, 8192])
        large_hi = 1 << rng.randint(15, 20)
        permille = rng.choice([20, 100, 300])
        small_hi = rng.randint(200, 2048)
        waves = rng.randint(2, 3)
        per = mean_request_bytes((16, small_hi), (8192, large_hi), permille)
        blocks = max(1, min(304, int(0.12 * heap * MIB / per / 256)))
        return {"kind": "frag", "heap_mib": heap, "blocks": blocks, "threads": 256, "waves": waves,
                "small_hi": small_hi, "large_lo": 8192, "large_hi": large_hi, "large_permille": permille}
    if kind == "batch":
        return {"kind": "batch", "heap_mib": rng.choice([8192, 16384]), "tuned": rng.random() < 0.5,
                "jobs": _log(rng, 8, 400), "tmin": 32, "tmax": _log(rng, 1024, 65536),
                "mean_size": rng.randint(24, 128), "max_size": 4096, "max_cycles": rng.randint(4, 16)}
    if kind == "serve":
        return {"kind": "serve", "heap_mib": rng.choice([16384, 32768, 65536]), "requests": _log(rng, 200, 6000),
                "median": rng.randint(200, 1024), "pipelined": rng.random() < 0.7}
    return {"kind": "slots", "heap_mib": _log(rng, 2048, 65536), "ops": rng.randint(100, 600)}


def _creation(case):
    return CreationPolicies.Scatter(pagesize=4096, accessblocksize=case["accessblock_mib"] * MIB, regionsize=16,
                                    wastefactor=2, resetfreedpages=bool(case.get("reset", False)))


def _stress_sizes(case, seed):
    """The table of a stress with table: uniform multiples of `step` in [lo, hi]."""
    n = (case["hi"] - case["lo"]) // case["step"] + 1
    rng = np.random.default_rng([seed, 1])
    count = case["blocks"] * case["threads"] * case["rounds"]
    if count > 1 << 22:  # one 2^20-entry draw, laid out again and again with other rotations
        base = rng.integers(0, n, size=1 << 20, dtype=np.int16)
        rows = -(-count // base.size)
        draws = np.concatenate([np.roll(base, int(s)) for s in rng.integers(0, base.size, size=rows)])[:count]
    else:
        draws = rng.integers(0, n, size=count, dtype=np.int16)
    return draws * np.int16(case["step"]) + np.int16(case["lo"])


def _live_sizes(case, seed):
    """Multiples of 4 bytes, as the verify workload's patterns are 4-byte words."""
    rng = np.random.default_rng([seed, 2])
    return rng.integers(case["lo"] // 4, case["hi"] // 4 + 1, size=case["blocks"] * case["threads"],
                        dtype=np.int32) * 4


def _slot_sizes(seed):
    """Sizes a program asks about: chunks of several classes, a page, a few multi-page blocks."""
    rng = np.random.default_rng([seed, 3])
    chunks = [16 * int(k) for k in rng.integers(1, 256, size=3)]
    return [16, 256] + chunks + [4096, 65536, 4096 * int(rng.integers(2, 300))]


def _requests(case, seed):
    return make_requests(case["requests"], 1e5, seed=seed, median=case["median"])


def prepare(case, seed):
    kind, heap = case["kind"], case["heap_mib"] * MIB
    st = {"case": case, "seed": seed, "kind": kind}
    if kind == "stress":
        dist = DistributionPolicies.XMallocSIMD(4096) if case["coalesce"] else DistributionPolicies.Noop()
        st["alloc"] = Allocator(_creation(case), dist, None, None, AlignmentPolicies.Shrink(16), size=heap)
        st["params"] = stress_params(case["blocks"], case["threads"], case["rounds"], case["lo"], case["hi"],
                                     case["step"], seed + 1, PATTERN_WARP if case["warp"] else PATTERN_THREAD)
        st["sizes"] = torch.from_numpy(_stress_sizes(case, seed)).cuda() if case["table"] else None
        st["stats"] = torch.zeros(4, dtype=torch.int64, device="cuda")
    elif kind == "live":
        st["alloc"] = Allocator(_creation(case), None, None, None, None, size=heap)
        st["sizes"] = torch.from_numpy(_live_sizes(case, seed)).cuda()
        st["offsets"] = torch.zeros(st["sizes"].numel(), dtype=torch.int64, device="cuda")
        st["errors"] = torch.zeros(1, dtype=torch.int64, device="cuda")
    elif kind == "frag":
        st["alloc"] = frag_allocator(heap, min(256 * MIB, heap // 2), GB300_FRAG_TUNED)
        per_wave = case["blocks"] * case["threads"]
        live = case["waves"] * per_wave
        half = np.random.default_rng([seed, 4]).permutation(live)[: live // 2].astype(np.int32)
        st["half"] = torch.from_numpy(half).cuda()
        st["every"] = torch.arange(live + per_wave, dtype=torch.int32, device="cuda")
        st["ptrs"] = torch.zeros(live + per_wave, dtype=torch.int64, device="cuda")
        st["sizes"] = torch.zeros(live + per_wave, dtype=torch.int32, device="cuda")
        small, large = (16, case["small_hi"]), (case["large_lo"], case["large_hi"])
        st["fill"] = frag_params(case["blocks"], case["threads"], seed + 1, 0, small, large, case["large_permille"],
                                 case["waves"])
        st["refill"] = frag_params(case["blocks"], case["threads"], seed + 1, live, small, large,
                                   case["large_permille"], 1)
        st["counters"] = torch.zeros(8, dtype=torch.int64, device="cuda")
    elif kind == "batch":
        if case["tuned"]:
            t = GB300_TUNED
            creation = CreationPolicies.Scatter(
                pagesize=t.pagesize, regionsize=t.regionsize, hashingK=t.hashingK, hashingDistMP=t.hashingDistMP,
                accessblocksize=_accessblock(heap, t.pagesize, t.accessblock_fraction))
            blocks = torch.cuda.get_device_properties(0).multi_processor_count * t.blocks_per_sm
        else:
            creation, blocks = CreationPolicies.Scatter(), 0
        st["alloc"] = Allocator(creation, DistributionPolicies.XMallocSIMD(creation.pagesize), None, None,
                                AlignmentPolicies.Shrink(16), size=heap)
        st["batch"] = Batch(st["alloc"], _jobs(case, seed), persistent_blocks=blocks)
    elif kind == "serve":
        creation = CreationPolicies.Scatter(pagesize=65536, accessblocksize=min(16384 * MIB, heap // 2),
                                            regionsize=16)
        st["alloc"] = Allocator(creation, DistributionPolicies.XMallocSIMD(65536), None, None,
                                AlignmentPolicies.Shrink(16), size=heap)
        st["server"] = Server(st["alloc"], slots=4096, max_chunks=128, step=64, queue_cap=8192)
        st["requests"] = _requests(case, seed)
    else:
        st["alloc"] = Allocator(CreationPolicies.Scatter(accessblocksize=512 * MIB), None, None, None, None,
                                size=heap)
        rng = np.random.default_rng([seed, 5])
        sizes = np.exp(rng.uniform(math.log(16), math.log(1 << 20), size=case["ops"])).astype(np.int64)
        ops = [("m", int(s)) for s in sizes]
        ops += [("f", int(i)) for i in rng.permutation(case["ops"])[: case["ops"] // 2]]
        run_program(st["alloc"], ops)
        st["slot_sizes"] = _slot_sizes(seed)
        st["out"] = torch.zeros(len(st["slot_sizes"]), dtype=torch.int32, device="cuda")
    return st


def _jobs(case, seed):
    return make_jobs(case["jobs"], seed=seed, tmin=case["tmin"], tmax=case["tmax"], mean_size=case["mean_size"],
                     max_size=case["max_size"], max_cycles=case["max_cycles"])


def run(st):
    kind, alloc, case = st["kind"], st["alloc"], st["case"]
    if kind == "stress":
        st["stats"].zero_()
        launch_stress(alloc, st["params"], st["sizes"].data_ptr() if st["sizes"] is not None else None,
                      st["stats"].data_ptr())
        return st["stats"]
    if kind == "batch":
        st["batch"].run()
        r = st["batch"].stats(clear=True).view(np.int64)
        return {"pairs": r[:, 0], "nulls": r[:, 1], "errors": r[:, 2], "checksum": r[:, 3]}
    if kind == "serve":
        r = st["server"].run(*st["requests"], realtime=False, pipelined=case["pipelined"])
        return {"checksum": r["checksum"].view(np.int64), "completed": r["completed"]}
    if kind == "slots":
        for k, size in enumerate(st["slot_sizes"]):
            alloc.getAvailableSlotsAsync(size, st["out"].data_ptr() + 4 * k)
        return st["out"]
    lib, stream = L.lib(), torch.cuda.current_stream().cuda_stream
    if kind == "live":
        st["errors"].zero_()
        args = (alloc.handle_ptr, case["blocks"], case["threads"], st["sizes"].data_ptr(), st["seed"] & 0xFFFF,
                st["offsets"].data_ptr())
        L.check(lib.mmc_run_alloc_offsets(*args, stream), "alloc_offsets")
        got = torch.where(st["offsets"] >= 0, st["sizes"], -1)  # what each thread holds
        L.check(lib.mmc_run_free_offsets(*args, st["errors"].data_ptr(), stream), "free_offsets")
        return {"sizes": got, "errors": st["errors"]}
    # frag
    st["counters"].zero_()
    ptrs, sizes, counters = (st[k].data_ptr() for k in ("ptrs", "sizes", "counters"))
    cap = st["ptrs"].numel()
    L.check(lib.mmc_run_fill(alloc.handle_ptr, ctypes.byref(st["fill"]), ptrs, sizes, cap, counters, stream), "fill")
    filled = st["counters"].clone()
    L.check(lib.mmc_run_free_list(alloc.handle_ptr, ptrs, sizes, st["half"].data_ptr(), st["half"].numel(), counters,
                                  stream), "free_list")
    L.check(lib.mmc_run_fill(alloc.handle_ptr, ctypes.byref(st["refill"]), ptrs, sizes, cap, counters, stream),
            "refill")
    L.check(lib.mmc_run_verify_list(alloc.handle_ptr, ptrs, sizes, cap, counters, stream), "verify_list")
    L.check(lib.mmc_run_free_list(alloc.handle_ptr, ptrs, sizes, st["every"].data_ptr(), cap, counters, stream),
            "free_list")
    return {"filled": filled, "end": st["counters"]}


def work(case):
    """Bytes each pass writes and reads: payload, tables and results, and the heap's words at the reference
    algorithm's count of atomics (three of 4 bytes for a malloc, two for a free) and 16 bytes of metadata reads."""
    kind, meta = case["kind"], 36
    if kind == "stress":
        pairs = case["blocks"] * case["threads"] * case["rounds"]
        return {"bytes": pairs * ((case["lo"] + case["hi"]) + meta + (2 if case["table"] else 0)) + 32, "flops": 0}
    if kind == "live":
        n = case["blocks"] * case["threads"]
        return {"bytes": n * ((case["lo"] + case["hi"]) + meta + 4 + 16 + 4), "flops": 0}
    if kind == "frag":
        n = (case["waves"] + 1) * case["blocks"] * case["threads"]
        pages = max(1.0, case["large_permille"] / 1000.0
                    * mean_request_bytes((16, case["small_hi"]), (case["large_lo"], case["large_hi"]), 1000) / 4096)
        return {"bytes": int(n * (meta + 24 + 16 * pages)), "flops": 0}
    if kind == "batch":
        threads = case["jobs"] * (case["tmax"] - case["tmin"]) / math.log(case["tmax"] / case["tmin"])
        pairs = threads * (1 + case["max_cycles"]) / 2
        return {"bytes": int(pairs * 2 * (case["mean_size"] + 8) + case["jobs"] * 72), "flops": 0}
    if kind == "serve":
        elements = case["requests"] * case["median"] * math.exp(0.5)
        return {"bytes": int(elements * 4 + case["requests"] * (24 + 16)), "flops": 0}
    pages = case["heap_mib"] * 256
    return {"bytes": pages * sum(8 if size < 4096 else 4 for size in _slot_sizes(0)), "flops": 0}


def exact(case, seed):
    """What follows from the inputs alone: every request is served, so the counts and the
    requests' checksums are known; a stress's and a batch's checksums follow from their pattern words alone
    and have no plain form."""
    kind = case["kind"]
    if kind == "live":
        return {"sizes": torch.from_numpy(_live_sizes(case, seed)), "errors": torch.zeros(1, dtype=torch.int64)}
    if kind == "serve":
        _, lengths, seeds = _requests(case, seed)
        sums = np.array([expected_checksum(int(s), int(n)) for s, n in zip(seeds, lengths)], dtype=np.uint64)
        return {"checksum": sums.view(np.int64), "completed": case["requests"]}
    if kind == "batch":
        zero = np.zeros(case["jobs"], dtype=np.int64)
        return {"pairs": expected_pairs(_jobs(case, seed)), "nulls": zero, "errors": zero, "checksum": None}
    return None
