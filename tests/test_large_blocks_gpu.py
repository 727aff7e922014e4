"""Kernels that call malloc in blocks of up to 1024 threads, without launch
bounds: the verify_heap tool and a user's kernel on the C++ handle API."""
import pytest

from tests.test_divergent_callers_gpu import churn
from tests.test_verify_heap_tool import _run_csv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [544, 768, 1024])
def test_verify_heap_with_large_blocks(threads):
    rc, v = _run_csv("--heapsize=1024", "--blocks=64", f"--threads={threads}")
    assert rc == 0 and v["correct"] == "1" and int(v["Blocksize"]) == threads, v
    assert int(v["usedSlots"]) > 0


@pytest.mark.parametrize("lo, hi", [(16, 600), (16, 6000)])
def test_user_kernel_of_1024_threads(lo, hi):
    (served, nulls, outside, wrong), flags = churn(76, 1024, 20, lo, hi)
    assert served > 76 * 1024
    assert (nulls, outside, wrong, flags) == (0, 0, 0, 0)
