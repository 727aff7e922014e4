"""A user's kernel (the C++ handle API, no launch bounds) whose threads allocate,
write, read back and free on schedules of their own, so the lanes of a warp come
to malloc and free in changing groups: every pointer lies in the pool, every
word reads back, no request fails. Sizes whose requests a warp joins, sizes of a
page's chunks, and a mix with multi-page requests; whole warps and a part."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def churn(blocks, threads, rounds, lo, hi):
    from mallocmc_gb300 import build

    ex = ctypes.CDLL(build.EXAMPLES_PATH)
    ex.mmcx_churn.argtypes = [ctypes.c_int] + [ctypes.c_uint] * 5 + [ctypes.c_void_p, ctypes.POINTER(ctypes.c_uint)]
    counts = np.zeros(4, dtype=np.uint64)
    flags = ctypes.c_uint()
    assert ex.mmcx_churn(0, blocks, threads, rounds, lo, hi, counts.ctypes.data, ctypes.byref(flags)) == 0
    return counts.tolist(), flags.value


@pytest.mark.parametrize("lo, hi", [(16, 112), (16, 1024), (200, 200), (16, 6000)])
@pytest.mark.parametrize("blocks, threads", [(1, 20), (5, 160), (304, 256)])
def test_every_group_gets_blocks_of_its_own(blocks, threads, lo, hi):
    (served, nulls, outside, wrong), flags = churn(blocks, threads, 40, lo, hi)
    assert served > blocks * threads
    assert (nulls, outside, wrong, flags) == (0, 0, 0, 0)
