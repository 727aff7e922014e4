/* cxx_examples.cu — user-side code written against the C++ drop-in API
 * (include/mallocMC/mallocMC.hpp), as the reference's examples are:
 *   example01  arrays of arrays allocated in kernels, vector addition, sums
 *              (reference: examples/mallocMC_example01.cpp)
 *   example03  device-side getAvailableSlots next to a live allocation
 *              (reference: examples/mallocMC_example03.cpp)
 * Built into libmallocmc_examples.so (linked against libmallocmc_gb300.so) and
 * driven by tests/test_cxx_api.py through the extern "C" wrappers below.
 *
 * Both reference examples construct a 1 GB heap with the default 2 GiB access
 * block; the reference divides by zero for that configuration
 * (Scatter.hpp:991-993). Here the same construction throws
 * std::invalid_argument, which mmcx_bad_config reports, and the examples run
 * with a 256 MiB access block.
 */
#include "mallocMC/mallocMC.hpp"

#include <cstdio>
#include <stdexcept>
#include <vector>

namespace
{
    struct ScatterHeapConfig
    {
        static constexpr auto pagesize = 4096;
        static constexpr auto accessblocksize = 256u * 1024u * 1024u;
        static constexpr auto regionsize = 16;
        static constexpr auto wastefactor = 2;
        static constexpr auto resetfreedpages = false;
    };
    struct ScatterHashConfig
    {
        static constexpr auto hashingK = 38183;
        static constexpr auto hashingDistMP = 17497;
        static constexpr auto hashingDistWP = 1;
        static constexpr auto hashingDistWPRel = 1;
    };
    struct ShrinkConfig
    {
        static constexpr auto dataAlignment = 16;
    };
    using Acc = mallocMC::AccGpuCuda;

    using ScatterAllocator = mallocMC::Allocator<
        Acc,
        mallocMC::CreationPolicies::Scatter<ScatterHeapConfig, ScatterHashConfig>,
        mallocMC::DistributionPolicies::Noop,
        mallocMC::OOMPolicies::ReturnNull,
        mallocMC::ReservePoolPolicies::AlpakaBuf<Acc>,
        mallocMC::AlignmentPolicies::Shrink<ShrinkConfig>>;

    using DefaultAllocator = mallocMC::Allocator<
        Acc,
        mallocMC::CreationPolicies::Scatter<>,
        mallocMC::DistributionPolicies::XMallocSIMD<>,
        mallocMC::OOMPolicies::ReturnNull,
        mallocMC::ReservePoolPolicies::AlpakaBuf<Acc>,
        mallocMC::AlignmentPolicies::Shrink<>>;

    using OldAllocator = mallocMC::Allocator<
        Acc,
        mallocMC::CreationPolicies::OldMalloc,
        mallocMC::DistributionPolicies::Noop,
        mallocMC::OOMPolicies::ReturnNull,
        mallocMC::ReservePoolPolicies::CudaSetLimits,
        mallocMC::AlignmentPolicies::Noop>;

    /* The reference's policy matrix (tests/policies.cpp:83-187): Scatter or
     * OldMalloc x XMallocSIMD or Noop x Shrink or Noop, each with its reserve
     * pool and ReturnNull; there one thread mallocs 4000 bytes and frees them. */
    template<class Creation, class Distribution, class ReservePool, class Alignment>
    using PolicyAllocator = mallocMC::Allocator<Acc, Creation, Distribution, mallocMC::OOMPolicies::ReturnNull,
                                                ReservePool, Alignment>;
    using Sc = mallocMC::CreationPolicies::Scatter<ScatterHeapConfig, ScatterHashConfig>;
    using Om = mallocMC::CreationPolicies::OldMalloc;
    using Xm = mallocMC::DistributionPolicies::XMallocSIMD<>;
    using Nd = mallocMC::DistributionPolicies::Noop;
    using Ab = mallocMC::ReservePoolPolicies::AlpakaBuf<Acc>;
    using Cl = mallocMC::ReservePoolPolicies::CudaSetLimits;
    using Sh = mallocMC::AlignmentPolicies::Shrink<ShrinkConfig>;
    using Na = mallocMC::AlignmentPolicies::Noop;

    template<class A>
    __global__ void policyMatrixKernel(typename A::AllocatorHandle h, int* ok)
    {
        const Acc acc{};
        void* p = h.malloc(acc, 4000);
        if(p != nullptr)
        {
            h.free(acc, p);
            *ok = 1;
        }
    }

    template<class A>
    std::string policy_info()
    {
        return A::info("\n");
    }

    __global__ void oldMallocKernel(OldAllocator::AllocatorHandle h, int length, unsigned long long* sums, int* fails)
    {
        const Acc acc{};
        const unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
        int* a = static_cast<int*>(h.malloc(acc, length * sizeof(int)));
        if(a == nullptr)
        {
            atomicAdd(fails, 1);
            sums[id] = 0;
            return;
        }
        unsigned long long s = 0;
        for(int i = 0; i < length; ++i)
            a[i] = static_cast<int>(id * length + i);
        for(int i = 0; i < length; ++i)
            s += static_cast<unsigned long long>(a[i]);
        sums[id] = s;
        if(h.getAvailableSlots(acc, 16) != 0u)
            atomicAdd(fails, 1000); /* OldMalloc provides no count: must be 0 */
        h.free(acc, a);
    }

    __device__ int** arA;
    __device__ int** arB;
    __device__ int** arC;
    __device__ int* ar3;

    __global__ void createArrayPointers(int x, int y, ScatterAllocator::AllocatorHandle h)
    {
        const Acc acc{};
        arA = static_cast<int**>(h.malloc(acc, sizeof(int*) * x * y));
        arB = static_cast<int**>(h.malloc(acc, sizeof(int*) * x * y));
        arC = static_cast<int**>(h.malloc(acc, sizeof(int*) * x * y));
    }

    __global__ void fillArrays(int length, ScatterAllocator::AllocatorHandle h, int* failures)
    {
        const Acc acc{};
        const unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
        arA[id] = static_cast<int*>(h.malloc(acc, length * sizeof(int)));
        arB[id] = static_cast<int*>(h.malloc(acc, length * sizeof(int)));
        arC[id] = static_cast<int*>(h.malloc(acc, length * sizeof(int)));
        if(!arA[id] || !arB[id] || !arC[id])
        {
            atomicAdd(failures, 1);
            return;
        }
        for(int i = 0; i < length; ++i)
        {
            arA[id][i] = static_cast<int>(id * length + i);
            arB[id][i] = static_cast<int>(id * length + i);
        }
    }

    __global__ void addArrays(int length, unsigned long long* sums)
    {
        const unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
        unsigned long long s = 0;
        if(arA[id] && arB[id] && arC[id])
            for(int i = 0; i < length; ++i)
            {
                arC[id][i] = arA[id][i] + arB[id][i];
                s += static_cast<unsigned long long>(arC[id][i]);
            }
        sums[id] = s;
    }

    __global__ void freeArrays(ScatterAllocator::AllocatorHandle h)
    {
        const unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
        h.free(arA[id]);
        h.free(arB[id]);
        h.free(arC[id]);
    }

    __global__ void freeArrayPointers(ScatterAllocator::AllocatorHandle h)
    {
        h.free(arA);
        h.free(arB);
        h.free(arC);
    }

    __global__ void example03Kernel(ScatterAllocator::AllocatorHandle h, unsigned* slots, int* values)
    {
        const Acc acc{};
        const unsigned id = threadIdx.x;
        if(id == 0)
            ar3 = static_cast<int*>(h.malloc(acc, sizeof(int) * 32));
        __syncthreads();
        slots[id] = h.getAvailableSlots(acc, 1);
        if(ar3 != nullptr)
        {
            ar3[id] = static_cast<int>(id);
            values[id] = ar3[id];
        }
        __syncthreads();
        if(id == 0)
            h.free(acc, ar3);
    }

    /* User code on the raw device API whose requests fit a page: the kernel
     * is built with SmallRequests, which leaves the multi-page search out of
     * it. Here one request above a page is made on purpose: it fails
     * (nullptr, MMC_DEVERR_PAGEBASED), while the same request through the
     * handle takes the multi-page path. */
    __global__ void smallRequestsKernel(ScatterAllocator::AllocatorHandle h, int* out)
    {
        using Small = mmc::dev::SmallRequests<ScatterAllocator::AllocatorHandle::Ids>;
        void* a = mmc::dev::malloc<Small>(h.devAllocator, 256);
        void* b = mmc::dev::malloc<Small>(h.devAllocator, 3 * 4096 + 16);
        void* c = h.malloc(3 * 4096 + 16);
        out[0] = a != nullptr;
        out[1] = b == nullptr;
        out[2] = c != nullptr;
        if(a != nullptr)
            mmc::dev::free<Small>(h.devAllocator, a);
        if(c != nullptr)
            h.free(c);
    }

    using ChurnAllocator = PolicyAllocator<Sc, Xm, Ab, Sh>;

    /* Threads that allocate, write, read back and free on schedules of their
     * own: a thread sits rounds out and keeps its block for some, so the lanes
     * of a warp come to malloc and free in changing groups. A pointer is used
     * only if its block lies inside the pool. counts: blocks served, NULLs,
     * pointers that are unaligned or outside the pool, words read back wrong. */
    __global__ void churnKernel(ChurnAllocator::AllocatorHandle h, unsigned rounds, unsigned lo, unsigned hi,
                                const char* pool, size_t pool_size, unsigned long long* counts)
    {
        const Acc acc{};
        const unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
        unsigned* held = nullptr;
        unsigned words = 0u, tag = 0u;
        for(unsigned r = 0; r <= rounds; ++r)
        {
            unsigned x = id * 2654435761u + r * 0x9E3779B9u;
            x = (x ^ (x >> 16)) * 0x85EBCA6Bu;
            x ^= x >> 13;
            if(held == nullptr && (x & 3u) != 0u && r < rounds)
            {
                const unsigned bytes = lo + (x >> 8) % (hi - lo + 1u);
                char* p = static_cast<char*>(h.malloc(acc, bytes));
                const size_t offset = static_cast<size_t>(p - pool);
                if(p == nullptr)
                    atomicAdd(&counts[1], 1ull);
                else if(offset >= pool_size || bytes > pool_size - offset || offset % ShrinkConfig::dataAlignment != 0u)
                    atomicAdd(&counts[2], 1ull);
                else
                {
                    atomicAdd(&counts[0], 1ull);
                    held = reinterpret_cast<unsigned*>(p);
                    words = bytes / 4u;
                    tag = x;
                    for(unsigned i = 0; i < words; ++i)
                        held[i] = tag + i;
                }
            }
            else if(held != nullptr && ((x & 4u) != 0u || r == rounds))
            {
                unsigned wrong = 0u;
                for(unsigned i = 0; i < words; ++i)
                    wrong += held[i] != tag + i ? 1u : 0u;
                if(wrong != 0u)
                    atomicAdd(&counts[3], static_cast<unsigned long long>(wrong));
                h.free(acc, held);
                held = nullptr;
            }
        }
    }

    /* Thread t asks for the free slots of sizes[t], `ahead` rounds of a loop
     * behind or ahead of its neighbours'. */
    __global__ void slotsOfSizesKernel(ScatterAllocator::AllocatorHandle h, const unsigned* sizes, unsigned ahead,
                                       unsigned* slots)
    {
        const Acc acc{};
        const unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
        for(unsigned r = 0; r <= (ahead != 0u ? id % ahead : 0u); ++r)
            slots[id] = h.getAvailableSlots(acc, sizes[id]);
    }

    /* Every thread asks for three pages, whole warps together, and marks the
     * first and last word; counts: blocks got, NULLs. */
    __global__ void threePagesKernel(ScatterAllocator::AllocatorHandle h, unsigned** blocks, unsigned* counts)
    {
        const Acc acc{};
        const unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
        unsigned* p = static_cast<unsigned*>(h.malloc(acc, 3 * 4096));
        blocks[id] = p;
        atomicAdd(&counts[p != nullptr ? 0 : 1], 1u);
        if(p != nullptr)
            p[0] = p[3 * 1024 - 1] = id;
    }

    __global__ void freeThreePagesKernel(ScatterAllocator::AllocatorHandle h, unsigned** blocks, unsigned* wrong)
    {
        const Acc acc{};
        const unsigned id = blockIdx.x * blockDim.x + threadIdx.x;
        unsigned* p = blocks[id];
        if(p == nullptr)
            return;
        if(p[0] != id || p[3 * 1024 - 1] != id)
            atomicAdd(wrong, 1u);
        h.free(acc, p);
    }

    /* Free pages that no multi-page search would find: their bits in the free-page
     * map are clear. */
    unsigned hidden_pages(const mmc_device_handle& d)
    {
        std::vector<uint32_t> sizes(d.numpages), map(d.numpages / 32u + 1u);
        cudaMemcpy(sizes.data(), d.chunksize, sizeof(uint32_t) * sizes.size(), cudaMemcpyDeviceToHost);
        cudaMemcpy(map.data(), d.freemap, sizeof(uint32_t) * map.size(), cudaMemcpyDeviceToHost);
        unsigned hidden = 0;
        for(uint32_t p = 0; p < d.numpages; ++p)
            hidden += sizes[p] == 0u && ((map[p / 32u] >> (p % 32u)) & 1u) == 0u ? 1u : 0u;
        return hidden;
    }

    int report(const std::exception& e)
    {
        std::fprintf(stderr, "mmcx: %s\n", e.what());
        return 1;
    }
} // namespace

extern "C" {

/* example01: returns 0 on success; *sum is the GPU sum of C = A + B over all
 * threads, *gaussian the closed form n(n-1) with n = threads * length,
 * *slots_1mib the host getAvailableSlots(1 MiB) before freeing. */
int mmcx_example01(int device, int length, unsigned long long* sum, unsigned long long* gaussian,
                   unsigned* slots_1mib, int* failures)
{
    try
    {
        cudaSetDevice(device);
        const unsigned block = 32;
        const unsigned grid = (length + block - 1) / block;
        ScatterAllocator alloc(device, nullptr, 1U * 1024U * 1024U * 1024U);
        int* d_fail = nullptr;
        unsigned long long* d_sums = nullptr;
        cudaMalloc(&d_fail, sizeof(int));
        cudaMemset(d_fail, 0, sizeof(int));
        cudaMalloc(&d_sums, sizeof(unsigned long long) * block * grid);
        createArrayPointers<<<1, 1>>>(grid, block, alloc.getAllocatorHandle());
        fillArrays<<<grid, block>>>(length, alloc.getAllocatorHandle(), d_fail);
        addArrays<<<grid, block>>>(length, d_sums);
        std::vector<unsigned long long> h(block * grid);
        cudaMemcpy(h.data(), d_sums, sizeof(unsigned long long) * h.size(), cudaMemcpyDeviceToHost);
        cudaMemcpy(failures, d_fail, sizeof(int), cudaMemcpyDeviceToHost);
        unsigned long long s = 0;
        for(auto v : h)
            s += v;
        *sum = s;
        const unsigned long long n = static_cast<unsigned long long>(block) * grid * length;
        *gaussian = n * (n - 1);
        if(mallocMC::Traits<ScatterAllocator>::providesAvailableSlots)
            *slots_1mib = alloc.getAvailableSlots(device, nullptr, 1024U * 1024U);
        freeArrays<<<grid, block>>>(alloc.getAllocatorHandle());
        freeArrayPointers<<<1, 1>>>(alloc.getAllocatorHandle());
        const cudaError_t e = cudaDeviceSynchronize();
        cudaFree(d_fail);
        cudaFree(d_sums);
        return e == cudaSuccess ? 0 : 2;
    }
    catch(const std::exception& e)
    {
        return report(e);
    }
}

/* example03: 32 threads of one block; slots[32] are the device-side counts of
 * 1-byte slots seen while thread 0's 128-byte block is live, values[32] what
 * each thread stored into it, *host_slots the host count after the free. */
int mmcx_example03(int device, unsigned* slots, int* values, unsigned* host_slots)
{
    try
    {
        cudaSetDevice(device);
        ScatterAllocator alloc(device, nullptr, 1U * 1024U * 1024U * 1024U);
        unsigned* d_slots = nullptr;
        int* d_values = nullptr;
        cudaMalloc(&d_slots, 32 * sizeof(unsigned));
        cudaMalloc(&d_values, 32 * sizeof(int));
        example03Kernel<<<1, 32>>>(alloc.getAllocatorHandle(), d_slots, d_values);
        cudaMemcpy(slots, d_slots, 32 * sizeof(unsigned), cudaMemcpyDeviceToHost);
        cudaMemcpy(values, d_values, 32 * sizeof(int), cudaMemcpyDeviceToHost);
        *host_slots = alloc.getAvailableSlots(device, nullptr, 1);
        cudaFree(d_slots);
        cudaFree(d_values);
        return cudaDeviceSynchronize() == cudaSuccess ? 0 : 2;
    }
    catch(const std::exception& e)
    {
        return report(e);
    }
}

/* The reference examples' configuration (1 GB heap, default 2 GiB access
 * block): returns 1 if construction throws std::invalid_argument, else 0.
 * No device work happens before the check. */
int mmcx_bad_config(int device)
{
    try
    {
        DefaultAllocator alloc(device, nullptr, 1U * 1024U * 1024U * 1024U);
        return 0;
    }
    catch(const std::invalid_argument&)
    {
        return 1;
    }
}

/* The same policy API over CUDA's own device heap (CreationPolicies::OldMalloc
 * with ReservePoolPolicies::CudaSetLimits): *sum over threads of their array
 * sums, *gaussian the closed form n(n-1)/2, host slot count (0: no count). */
int mmcx_oldmalloc(int device, int length, unsigned long long* sum, unsigned long long* gaussian, unsigned* slots,
                   int* failures)
{
    try
    {
        cudaSetDevice(device);
        OldAllocator alloc(device, nullptr, 64U * 1024U * 1024U);
        const unsigned block = 64, grid = 8;
        int* d_fail = nullptr;
        unsigned long long* d_sums = nullptr;
        cudaMalloc(&d_fail, sizeof(int));
        cudaMemset(d_fail, 0, sizeof(int));
        cudaMalloc(&d_sums, sizeof(unsigned long long) * block * grid);
        oldMallocKernel<<<grid, block>>>(alloc.getAllocatorHandle(), length, d_sums, d_fail);
        std::vector<unsigned long long> h(block * grid);
        cudaMemcpy(h.data(), d_sums, sizeof(unsigned long long) * h.size(), cudaMemcpyDeviceToHost);
        cudaMemcpy(failures, d_fail, sizeof(int), cudaMemcpyDeviceToHost);
        unsigned long long s = 0;
        for(auto v : h)
            s += v;
        *sum = s;
        const unsigned long long n = static_cast<unsigned long long>(block) * grid * length;
        *gaussian = n * (n - 1) / 2;
        *slots = alloc.getAvailableSlots(device, nullptr, 16);
        const cudaError_t e = cudaDeviceSynchronize();
        cudaFree(d_fail);
        cudaFree(d_sums);
        return e == cudaSuccess ? 0 : 2;
    }
    catch(const std::exception& e)
    {
        return report(e);
    }
}

/* Threads on schedules of their own (churnKernel) over a 1 GiB heap: counts[4]
 * = {blocks served, NULLs, bad pointers, wrong words}, *flags the heap's device
 * error bits. 3: the launch was refused. */
int mmcx_churn(int device, unsigned blocks, unsigned threads, unsigned rounds, unsigned lo, unsigned hi,
               unsigned long long* counts, unsigned* flags)
{
    try
    {
        cudaSetDevice(device);
        ChurnAllocator alloc(device, nullptr, 1U * 1024U * 1024U * 1024U);
        const auto pool = alloc.getHeapLocations().at(0);
        unsigned long long* d_counts = nullptr;
        cudaMalloc(&d_counts, 4 * sizeof(unsigned long long));
        cudaMemset(d_counts, 0, 4 * sizeof(unsigned long long));
        churnKernel<<<blocks, threads>>>(alloc.getAllocatorHandle(), rounds, lo, hi, static_cast<const char*>(pool.p),
                                         pool.size, d_counts);
        const bool refused = cudaGetLastError() != cudaSuccess;
        cudaMemcpy(counts, d_counts, 4 * sizeof(unsigned long long), cudaMemcpyDeviceToHost);
        *flags = alloc.errorFlags();
        cudaFree(d_counts);
        return refused ? 3 : (cudaDeviceSynchronize() == cudaSuccess ? 0 : 2);
    }
    catch(const std::exception& e)
    {
        return report(e);
    }
}

/* The same, `times` launches on one heap; *hidden: free pages hidden at the end,
 * all blocks freed. */
int mmcx_churn_map(int device, unsigned times, unsigned blocks, unsigned threads, unsigned lo, unsigned hi,
                   unsigned long long* counts, unsigned* hidden)
{
    try
    {
        cudaSetDevice(device);
        ChurnAllocator alloc(device, nullptr, 1U * 1024U * 1024U * 1024U);
        const auto pool = alloc.getHeapLocations().at(0);
        unsigned long long* d_counts = nullptr;
        cudaMalloc(&d_counts, 4 * sizeof(unsigned long long));
        cudaMemset(d_counts, 0, 4 * sizeof(unsigned long long));
        for(unsigned i = 0; i < times; ++i)
            churnKernel<<<blocks, threads>>>(alloc.getAllocatorHandle(), 20u + i, lo, hi,
                                             static_cast<const char*>(pool.p), pool.size, d_counts);
        cudaMemcpy(counts, d_counts, 4 * sizeof(unsigned long long), cudaMemcpyDeviceToHost);
        *hidden = hidden_pages(alloc.getAllocatorHandle().devAllocator);
        cudaFree(d_counts);
        return cudaDeviceSynchronize() == cudaSuccess ? 0 : 2;
    }
    catch(const std::exception& e)
    {
        return report(e);
    }
}

/* Device-side slot counts of n sizes (n a multiple of 32), a thread each, on a
 * heap partly used, and the host's counts of the same sizes. */
int mmcx_slots_of_sizes(int device, const unsigned* sizes, unsigned n, unsigned ahead, unsigned* slots, unsigned* host)
{
    try
    {
        cudaSetDevice(device);
        ScatterAllocator alloc(device, nullptr, 300U * 1024U * 1024U);
        unsigned** d_blocks = nullptr;
        unsigned *d_counts = nullptr, *d_sizes = nullptr, *d_slots = nullptr;
        cudaMalloc(&d_blocks, sizeof(unsigned*) * 96);
        cudaMalloc(&d_counts, 2 * sizeof(unsigned));
        cudaMalloc(&d_sizes, sizeof(unsigned) * n);
        cudaMalloc(&d_slots, sizeof(unsigned) * n);
        threePagesKernel<<<1, 96>>>(alloc.getAllocatorHandle(), d_blocks, d_counts);
        cudaMemcpy(d_sizes, sizes, sizeof(unsigned) * n, cudaMemcpyHostToDevice);
        slotsOfSizesKernel<<<n / 32u, 32>>>(alloc.getAllocatorHandle(), d_sizes, ahead, d_slots);
        cudaMemcpy(slots, d_slots, sizeof(unsigned) * n, cudaMemcpyDeviceToHost);
        for(unsigned i = 0; i < n; ++i)
            host[i] = alloc.getAvailableSlots(device, nullptr, sizes[i]);
        cudaFree(d_blocks);
        cudaFree(d_counts);
        cudaFree(d_sizes);
        cudaFree(d_slots);
        return cudaDeviceSynchronize() == cudaSuccess ? 0 : 2;
    }
    catch(const std::exception& e)
    {
        return report(e);
    }
}

/* Multi-page requests of 256 threads, twice, on a heap whose service is left by
 * the host as a warp that gave up might leave it: 0: locked by nobody who
 * serves; 1: a ticket drawn and never written; 2: a request given up, which a
 * server passes; 3: untouched. out[6] = {blocks got, NULLs (both times), words
 * wrong, whether the service is closed, pages still claimed, device error bits}. */
int mmcx_service_wait(int device, int state, unsigned* out)
{
    try
    {
        cudaSetDevice(device);
        ScatterAllocator alloc(device, nullptr, 1U * 1024U * 1024U * 1024U);
        const auto handle = alloc.getAllocatorHandle();
        const mmc_device_handle& d = handle.devAllocator;
        mmc_page_service* service = mmc::dev::page_service(d.state);
        const unsigned one = 1u, gone = mmc::dev::kPageGone | 3u;
        if(state == 0)
            cudaMemcpy(&service->lock, &one, sizeof(one), cudaMemcpyHostToDevice);
        if(state == 1 || state == 2)
            cudaMemcpy(&service->tail, &one, sizeof(one), cudaMemcpyHostToDevice);
        if(state == 2)
            cudaMemcpy(&service->ring[0], &gone, sizeof(gone), cudaMemcpyHostToDevice);
        const unsigned threads = 64, grid = 4;
        unsigned** d_blocks = nullptr;
        unsigned* d_counts = nullptr;
        cudaMalloc(&d_blocks, sizeof(unsigned*) * threads * grid);
        cudaMalloc(&d_counts, 3 * sizeof(unsigned));
        cudaMemset(d_counts, 0, 3 * sizeof(unsigned));
        for(int again = 0; again < 2; ++again)
        {
            threePagesKernel<<<grid, threads>>>(handle, d_blocks, d_counts);
            freeThreePagesKernel<<<grid, threads>>>(handle, d_blocks, d_counts + 2);
        }
        cudaMemcpy(out, d_counts, 3 * sizeof(unsigned), cudaMemcpyDeviceToHost);
        cudaMemcpy(out + 3, &service->closed, sizeof(unsigned), cudaMemcpyDeviceToHost);
        std::vector<uint32_t> chunksizes(d.numpages);
        cudaMemcpy(chunksizes.data(), d.chunksize, sizeof(uint32_t) * d.numpages, cudaMemcpyDeviceToHost);
        out[4] = 0u;
        for(const uint32_t c : chunksizes)
            out[4] += c != 0u ? 1u : 0u;
        out[5] = alloc.errorFlags();
        cudaFree(d_blocks);
        cudaFree(d_counts);
        return cudaDeviceSynchronize() == cudaSuccess ? 0 : 2;
    }
    catch(const std::exception& e)
    {
        return report(e);
    }
}

/* SmallRequests: out[3] = {the small request succeeded, the request above a
 * page failed, the same request through the handle succeeded}; *flags the
 * heap's device error bits afterwards. */
int mmcx_small_requests(int device, int* out, unsigned* flags)
{
    try
    {
        cudaSetDevice(device);
        ScatterAllocator alloc(device, nullptr, 1U * 1024U * 1024U * 1024U);
        int* d_out = nullptr;
        cudaMalloc(&d_out, 3 * sizeof(int));
        smallRequestsKernel<<<1, 1>>>(alloc.getAllocatorHandle(), d_out);
        cudaMemcpy(out, d_out, 3 * sizeof(int), cudaMemcpyDeviceToHost);
        *flags = alloc.errorFlags();
        cudaFree(d_out);
        return cudaDeviceSynchronize() == cudaSuccess ? 0 : 2;
    }
    catch(const std::exception& e)
    {
        return report(e);
    }
}

/* info() strings of the two allocator types (host only). */
/* The info() strings of the eight allocators of the reference's policy matrix,
 * separated by "--" lines (host only). */
int mmcx_policy_matrix_info(char* buf, size_t len)
{
    const std::string s = policy_info<PolicyAllocator<Sc, Xm, Ab, Sh>>() + "--\n"
                          + policy_info<PolicyAllocator<Sc, Xm, Ab, Na>>() + "--\n"
                          + policy_info<PolicyAllocator<Sc, Nd, Ab, Sh>>() + "--\n"
                          + policy_info<PolicyAllocator<Sc, Nd, Ab, Na>>() + "--\n"
                          + policy_info<PolicyAllocator<Om, Xm, Cl, Sh>>() + "--\n"
                          + policy_info<PolicyAllocator<Om, Xm, Cl, Na>>() + "--\n"
                          + policy_info<PolicyAllocator<Om, Nd, Cl, Sh>>() + "--\n"
                          + policy_info<PolicyAllocator<Om, Nd, Cl, Na>>();
    if(buf == nullptr || len == 0)
        return 1;
    std::snprintf(buf, len, "%s", s.c_str());
    return s.size() < len ? 0 : 1;
}

/* The device code of the same eight allocators, compiled: the host entry of
 * each one's malloc(4000)/free kernel (i in 0..7, in the order above). */
const void* mmcx_policy_matrix_kernel(int i)
{
    static const void* const k[8] = {
        reinterpret_cast<const void*>(&policyMatrixKernel<PolicyAllocator<Sc, Xm, Ab, Sh>>),
        reinterpret_cast<const void*>(&policyMatrixKernel<PolicyAllocator<Sc, Xm, Ab, Na>>),
        reinterpret_cast<const void*>(&policyMatrixKernel<PolicyAllocator<Sc, Nd, Ab, Sh>>),
        reinterpret_cast<const void*>(&policyMatrixKernel<PolicyAllocator<Sc, Nd, Ab, Na>>),
        reinterpret_cast<const void*>(&policyMatrixKernel<PolicyAllocator<Om, Xm, Cl, Sh>>),
        reinterpret_cast<const void*>(&policyMatrixKernel<PolicyAllocator<Om, Xm, Cl, Na>>),
        reinterpret_cast<const void*>(&policyMatrixKernel<PolicyAllocator<Om, Nd, Cl, Sh>>),
        reinterpret_cast<const void*>(&policyMatrixKernel<PolicyAllocator<Om, Nd, Cl, Na>>)};
    return (i >= 0 && i < 8) ? k[i] : nullptr;
}

int mmcx_info(char* buf, size_t len)
{
    const std::string s = ScatterAllocator::info("\n") + "--\n" + DefaultAllocator::info("\n");
    if(buf == nullptr || len == 0)
        return 1;
    const size_t n = std::min(len - 1, s.size());
    std::copy(s.begin(), s.begin() + static_cast<long>(n), buf);
    buf[n] = '\0';
    return 0;
}

} /* extern "C" */
