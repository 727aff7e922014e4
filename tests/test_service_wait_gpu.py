"""The multi-page service when a wait runs out: its requests and all later ones are
served without it, the error bit says so once, and nothing stays claimed. A
request given up is passed by the server. The waits end by themselves, in seconds."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LOCKED, HOLE, GIVEN_UP, UNTOUCHED = range(4)


@pytest.mark.parametrize("state", [UNTOUCHED, GIVEN_UP, LOCKED, HOLE])
def test_requests_are_served_when_a_wait_runs_out(state):
    from mallocmc_gb300 import _lib as L
    from mallocmc_gb300 import build

    ex = ctypes.CDLL(build.EXAMPLES_PATH)
    ex.mmcx_service_wait.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_void_p]
    out = np.zeros(6, dtype=np.uint32)
    assert ex.mmcx_service_wait(0, state, out.ctypes.data) == 0
    got, nulls, wrong, closed, claimed, flags = out.tolist()
    assert (got, nulls, wrong, claimed) == (2 * 256, 0, 0, 0)
    assert closed == (1 if state in (LOCKED, HOLE) else 0)
    assert flags == (L.MMC_DEVERR_TIMEOUT if state in (LOCKED, HOLE) else 0)
