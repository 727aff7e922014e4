"""What malloc and free cost a user's kernel in registers, as ptxas reports it for
kernels without launch bounds: 64 at most, so blocks of 1024 threads launch and
four blocks of 256 share an SM, and nothing spilled."""
import re
import subprocess

import pytest

KERNELS = """
#include <mallocMC/scatter_device.cuh>
using namespace mmc::dev;
template<class Ids>
__global__ void one(mmc_device_handle h, void** p, size_t bytes)
{
    p[blockIdx.x * blockDim.x + threadIdx.x] = mmc::dev::malloc<Ids>(h, bytes + threadIdx.x);
}
template<class Ids>
__global__ void rounds(mmc_device_handle h, unsigned n, size_t bytes)
{
    for(unsigned r = 0; r < n; ++r)
    {
        auto* p = static_cast<volatile unsigned*>(mmc::dev::malloc<Ids>(h, bytes + r + threadIdx.x));
        if(p == nullptr)
            continue;
        *p = r;
        mmc::dev::free<Ids>(h, const_cast<unsigned*>(p));
    }
}
template __global__ void one<%(ids)s>(mmc_device_handle, void**, size_t);
template __global__ void rounds<%(ids)s>(mmc_device_handle, unsigned, size_t);
"""


@pytest.mark.parametrize("ids", ["GpuIds", "GpuIdsDefault", "SmallRequests<GpuIdsDefault>"])
def test_registers_of_a_user_kernel(tmp_path, ids):
    from mallocmc_gb300 import build

    src = tmp_path / "user.cu"
    src.write_text(KERNELS % {"ids": ids})
    cmd = [build.nvcc()] + build.ARCH + ["-O3", "-std=c++17", "--expt-relaxed-constexpr", "-I" + build.INCLUDE,
                                         "-Xptxas", "-v", "-c", str(src), "-o", str(tmp_path / "user.o")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    used = [int(n) for n in re.findall(r"Used (\d+) registers", r.stdout + r.stderr)]
    assert len(used) == 2 and max(used) <= 64, used
    spills = [int(n) for n in re.findall(r"(\d+) bytes spill", r.stdout + r.stderr)]
    assert spills and max(spills) == 0
