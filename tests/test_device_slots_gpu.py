"""Device-side slot counts by lanes that ask for different sizes at one call, below
and above a page, and from different rounds of one loop: each gets the count the
host gets for its size."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ahead", [0, 3])
@pytest.mark.parametrize("kind", ["one", "small", "pages", "mixed"])
def test_lanes_with_sizes_of_their_own(kind, ahead):
    from mallocmc_gb300 import build

    ex = ctypes.CDLL(build.EXAMPLES_PATH)
    ex.mmcx_slots_of_sizes.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_uint, ctypes.c_uint, ctypes.c_void_p,
                                       ctypes.c_void_p]
    rng = np.random.default_rng(len(kind))
    n = 64
    choices = {"one": [20000], "small": [16, 64, 500, 2048, 4095], "pages": [4096, 4097, 9000, 40000, 1 << 20],
               "mixed": [1, 64, 3000, 4096, 5000, 100000]}[kind]
    sizes = rng.choice(choices, size=n).astype(np.uint32)
    slots, host = np.zeros(n, dtype=np.uint32), np.zeros(n, dtype=np.uint32)
    assert ex.mmcx_slots_of_sizes(0, sizes.ctypes.data, n, ahead, slots.ctypes.data, host.ctypes.data) == 0
    assert np.array_equal(slots, host)
    assert host.min() > 0
