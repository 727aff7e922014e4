"""Multi-page requests of whole and parted warps while other warps free theirs: in
the end every free page has its bit in the free-page map, so none is lost to later
searches."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks, threads, lo, hi", [(152, 96, 3000, 24000), (304, 256, 4096, 12288),
                                                     (76, 1024, 64, 9000)])
def test_no_free_page_is_hidden(blocks, threads, lo, hi):
    from mallocmc_gb300 import build

    ex = ctypes.CDLL(build.EXAMPLES_PATH)
    ex.mmcx_churn_map.argtypes = [ctypes.c_int] + [ctypes.c_uint] * 5 + [ctypes.c_void_p, ctypes.POINTER(ctypes.c_uint)]
    counts = np.zeros(4, dtype=np.uint64)
    hidden = ctypes.c_uint()
    assert ex.mmcx_churn_map(0, 12, blocks, threads, lo, hi, counts.ctypes.data, ctypes.byref(hidden)) == 0
    served, _, outside, wrong = counts.tolist()
    assert served > 0 and outside == 0 and wrong == 0
    assert hidden.value == 0
