/* Internal helpers shared by the translation units of libmallocmc_gb300.so. */
#pragma once

#include "mallocmc_gb300.h"
#include "mallocMC/scatter_device.cuh"

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include <string>

/* Run the statements in __VA_ARGS__ with `Ids` naming the thread-id type the
 * heap's kernels are launched with: GpuIdsDefault (the policy values fixed at
 * compile time) when the handle holds the default configuration, GpuIds (read
 * from the handle) otherwise. */
#define MMC_DISPATCH_IDS(handle, ...)                                                                                 \
    do                                                                                                                 \
    {                                                                                                                  \
        if(mmc::dev::GpuIdsDefault::matches(handle))                                                                   \
        {                                                                                                              \
            using Ids = mmc::dev::GpuIdsDefault;                                                                       \
            __VA_ARGS__;                                                                                               \
        }                                                                                                              \
        else                                                                                                           \
        {                                                                                                              \
            using Ids = mmc::dev::GpuIds;                                                                              \
            __VA_ARGS__;                                                                                               \
        }                                                                                                              \
    } while(0)

/* As MMC_DISPATCH_IDS, for a launch whose largest request (bytes, before
 * padding) the host knows: when it fits a page after padding, the default
 * configuration's instance is the one without the multi-page path
 * (mmc::dev::SmallRequests). */
#define MMC_DISPATCH_IDS_SIZED(handle, max_request, ...)                                                              \
    do                                                                                                                 \
    {                                                                                                                  \
        if(mmc::dev::GpuIdsDefault::matches(handle))                                                                   \
        {                                                                                                              \
            if(mmc::dev::apply_padding(16u, (max_request)) <= (handle).pagesize)                                      \
            {                                                                                                          \
                using Ids = mmc::dev::SmallRequests<mmc::dev::GpuIdsDefault>;                                          \
                __VA_ARGS__;                                                                                           \
            }                                                                                                          \
            else                                                                                                       \
            {                                                                                                          \
                using Ids = mmc::dev::GpuIdsDefault;                                                                   \
                __VA_ARGS__;                                                                                           \
            }                                                                                                          \
        }                                                                                                              \
        else                                                                                                           \
        {                                                                                                              \
            using Ids = mmc::dev::GpuIds;                                                                              \
            __VA_ARGS__;                                                                                               \
        }                                                                                                              \
    } while(0)

namespace mmc
{
    namespace host
    {
        /* Record msg as the calling thread's last error and return st. */
        mmc_status fail(mmc_status st, const std::string& msg);
        /* If e is an error: record it (with what) and return MMC_ERR_CUDA. */
        mmc_status cuda_check(cudaError_t e, const char* what);

        inline cudaStream_t as_stream(void* s) { return static_cast<cudaStream_t>(s); }

        /* For kernels launched by launch_after: let the stream's next such
         * kernel come in, and wait until the one before has ended and its
         * writes are visible. First thing in the kernel. */
        __device__ __forceinline__ void await_previous()
        {
            asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
            asm volatile("griddepcontrol.wait;" ::: "memory");
        }

        /* Launch a kernel whose blocks may come in before the stream's last
         * kernel has ended (programmatic stream serialisation); it waits for
         * that itself (await_previous), so only the launch overlaps. */
        template<class... Params, class... Args>
        cudaError_t launch_after(void (*kernel)(Params...), unsigned grid, unsigned block, cudaStream_t s, Args... args)
        {
            cudaLaunchAttribute attr{};
            attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr.val.programmaticStreamSerializationAllowed = 1;
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(grid);
            cfg.blockDim = dim3(block);
            cfg.stream = s;
            cfg.attrs = &attr;
            cfg.numAttrs = 1;
            return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
        }

        /* This thread's share of the free slots of size slot < pagesize on pages
         * [b0, b1), b0 a multiple of 4, of a block of nthreads threads: the
         * single-page branch of getAvailaibleSlotsDeviceFunction
         * (Scatter.hpp:1164-1193). Chunk sizes and fill counts are read with
         * 16-byte loads, four pages of both per load, two such pairs in
         * flight; an array that starts off a 16-byte boundary is read word by
         * word. */
        __device__ __forceinline__ uint32_t free_slots_of_range(const mmc_device_handle& h, uint32_t slot, uint32_t b0,
                                                                uint32_t b1, uint32_t nthreads)
        {
            const uint32_t maxchunksize = dev::umin(h.pagesize, h.wastefactor * slot);
            const uint32_t slotChunk = dev::umax(slot, h.paddedMinChunkSize);
            const uint32_t cap = dev::page_capacity(h, slotChunk);
            const bool aligned
                = ((reinterpret_cast<uintptr_t>(h.chunksize) | reinterpret_cast<uintptr_t>(h.count)) & 15u) == 0u;
            const uint32_t quads = aligned ? (b1 - b0) / 4u : 0u; /* b1 >= b0 */
            const uint4* cs = reinterpret_cast<const uint4*>(h.chunksize + b0);
            const uint4* ct = reinterpret_cast<const uint4*>(h.count + b0);
            uint32_t sum = 0u;
            for(uint32_t q = threadIdx.x; q < quads; q += 2u * nthreads)
            {
                uint4 v[2], c[2];
#pragma unroll
                for(uint32_t k = 0; k < 2u; ++k)
                {
                    const bool in = q + k * nthreads < quads;
                    v[k] = in ? __ldcg(cs + q + k * nthreads) : make_uint4(~0u, ~0u, ~0u, ~0u);
                    c[k] = in ? __ldcg(ct + q + k * nthreads) : make_uint4(0u, 0u, 0u, 0u);
                }
#pragma unroll
                for(uint32_t k = 0; k < 2u; ++k)
                {
                    const uint32_t w[4] = {v[k].x, v[k].y, v[k].z, v[k].w}, n[4] = {c[k].x, c[k].y, c[k].z, c[k].w};
#pragma unroll
                    for(uint32_t j = 0; j < 4u; ++j)
                        if(w[j] >= slot && w[j] <= maxchunksize)
                            sum += (w[j] == slotChunk ? cap : dev::page_capacity(h, w[j])) - n[j];
                        else if(w[j] == 0u)
                            sum += cap - n[j];
                }
            }
            for(uint32_t pg = b0 + 4u * quads + threadIdx.x; pg < b1; pg += nthreads)
                sum += dev::page_free_slots(h, __ldcg(&h.chunksize[pg]), __ldcg(&h.count[pg]), slot, maxchunksize,
                                            slotChunk, cap);
            return sum;
        }

        /* Grid for whole-heap scans: a multiple of the SM count. */
        unsigned scan_grid(int device);

        /* Launch the two-pass free-slot count of `slot` (already padded) and
         * leave the unsigned result in *result_dev (device memory). */
        mmc_status launch_available_slots(mmc_heap* heap, uint32_t slot, cudaStream_t s, unsigned* result_dev);

        /* Device-side word that receives the result of mmc_available_slots. */
        unsigned* slots_result_word(mmc_heap* heap);

        /* An NVTX range over a host entry point's work (heap set-up, slot
         * counts, launches of the batched and serving kernels), so Nsight
         * tools show each phase by name; without a tool attached it costs a
         * call into an empty stub. */
        struct NvtxRange
        {
            explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
            ~NvtxRange() { nvtxRangePop(); }
            NvtxRange(const NvtxRange&) = delete;
            NvtxRange& operator=(const NvtxRange&) = delete;
        };
    } // namespace host
} // namespace mmc
