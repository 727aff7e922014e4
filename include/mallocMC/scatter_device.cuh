/* scatter_device.cuh — device side of the GB300 ScatterAlloc heap.
 *
 * Header-only __device__ code: user kernels include it (directly or through
 * <mallocMC/mallocMC.hpp>) and call malloc/free/getAvailableSlots inline, as
 * with the reference's AllocatorHandleImpl (mallocMC_allocator_handle.hpp:35-63).
 * The algorithm is the reference's ScatterAlloc
 * (src/include/mallocMC/creationPolicies/Scatter.hpp); every function cites the
 * lines it follows. What is GB300-specific:
 *   - the handle carries every immutable heap field by value (kernel parameter
 *     space), so only the mutable words are read from memory;
 *   - the page-table entries are three word arrays (chunksize[], count[],
 *     bitmask[]) instead of an array of 12-byte structs: same bytes, same
 *     numpages, but scans read only the words they need, fully coalesced;
 *   - relaxed device-scope atomics (atom/red .relaxed.gpu) on L2-resident words
 *     and ld.relaxed.gpu for the racy metadata reads;
 *   - XMallocSIMD's warp coalescing uses __ballot_sync/__shfl_sync over the
 *     lanes that are active at the call, not shared-memory counters;
 *   - every spin is bounded: the page-based mutex gives up after a fixed
 *     number of backed-off tries, records MMC_DEVERR_TIMEOUT and returns NULL;
 *     a wait for the multi-page service ends in the lock-free search; the
 *     bit-claim retry loop gives up after MMC_USESPOT_MAX_TRIES.
 * Thread-id sources are a template parameter: GpuIds reads %laneid/%warpid/
 * %smid (mallocMC_utils.hpp:91-150); SerialIds is the reference CPU backend
 * (all zero, warp size 1), which makes one device thread reproduce the
 * reference's CPU-serial allocation sequence bit for bit.
 */
#pragma once

#include "../mallocmc_gb300.h"

#include <cstdint>

#ifndef MMC_USESPOT_MAX_TRIES
#define MMC_USESPOT_MAX_TRIES 256u
#endif
#ifndef MMC_MUTEX_MAX_SPINS
#define MMC_MUTEX_MAX_SPINS (1u << 22)
#endif
/* looks at the multi-page service without a ticket served, one to two
 * microseconds each (a batch reads the heap's free-page bitmap twice at most) */
#ifndef MMC_SERVICE_MAX_IDLE
#define MMC_SERVICE_MAX_IDLE (1u << 20)
#endif

/* Mutable heap words, each on its own 128-byte line. */
struct mmc_heap_state
{
    uint32_t pagebasedMutex; /* Scatter.hpp:269 */
    uint32_t pad0[31];
    uint32_t firstFreePageBased; /* Scatter.hpp:270 */
    uint32_t pad1[31];
    uint32_t firstfreeblock; /* Scatter.hpp:271 */
    uint32_t pad2[31];
    uint32_t error_flags; /* MMC_DEVERR_* */
    uint32_t pad3[31];
    /* event counters, maintained only in builds with MMC_DEVICE_STATS (MMC_STAT_*) */
    unsigned long long stats[16];
};

/* Multi-page requests of whole warps waiting to be served (see
 * page_service_run): a ring of tickets. It follows mmc_heap_state in the
 * heap's device block. */
#define MMC_PAGE_RING 32768u
struct mmc_page_service
{
    uint32_t lock; /* held by the warp that serves */
    uint32_t closed; /* set when a wait ran out: requests take the lock-free search */
    uint32_t pad0[30];
    uint32_t tail; /* tickets handed out */
    uint32_t pad1[31];
    uint32_t head; /* tickets served; the lock's holder moves it */
    uint32_t pad2[31];
    uint32_t ring[MMC_PAGE_RING]; /* 0: idle; kPageAsk or kPageGone | pages; kPageAnswer | page */
};

#ifdef MMC_DEVICE_STATS
#define MMC_STAT(h, i) atomicAdd(&(h).state->stats[(i)], 1ull)
#define MMC_STAT_ADD(h, i, n) atomicAdd(&(h).state->stats[(i)], static_cast<unsigned long long>(n))
#else
#define MMC_STAT(h, i) ((void) 0)
#define MMC_STAT_ADD(h, i, n) ((void) 0)
#endif

namespace mmc
{
    namespace dev
    {
        using u32 = uint32_t;
        using u64 = uint64_t;

        /* ---------------------------------------------------------- thread ids */
        struct GpuIds
        {
            static constexpr u32 warpSize = 32u; /* mallocMC_utils.hpp:72-73 */
            static constexpr bool coalesce = true;
            /* read the racy first-free-block hint through L1 (it changes rarely
             * and a stale value only moves where the search starts) */
            static constexpr bool cachedHints = true;
            /* requests above a page take the multi-page path (SmallRequests
             * leaves it out) */
            static constexpr bool pageBased = true;
            __device__ static __forceinline__ u32 laneid()
            {
                u32 r;
                asm volatile("mov.u32 %0, %%laneid;" : "=r"(r));
                return r;
            }
            __device__ static __forceinline__ u32 warpid()
            {
                u32 r;
                asm volatile("mov.u32 %0, %%warpid;" : "=r"(r));
                return r;
            }
            __device__ static __forceinline__ u32 smid()
            {
                u32 r;
                asm volatile("mov.u32 %0, %%smid;" : "=r"(r));
                return r;
            }
            /* the heap's policy values, read from the handle at run time */
            __device__ static __forceinline__ u32 reset(const mmc_device_handle& h) { return h.resetfreedpages; }
            __device__ static __forceinline__ u32 distribution(const mmc_device_handle& h) { return h.distribution; }
            __device__ static __forceinline__ u32 oom(const mmc_device_handle& h) { return h.oom_policy; }
            __device__ static __forceinline__ u32 alignment(const mmc_device_handle& h) { return h.dataAlignment; }
        };

        /* GpuIds with the policy values fixed at compile time, as the
         * reference's template parameters fix them (Scatter's resetfreedpages,
         * the distribution, OOM and alignment policies): code for the other
         * values drops out of the kernel, which shortens the malloc and free
         * paths the instruction cache holds (ncu counts instruction-fetch
         * stalls as the stress and batched kernels' top stall; 6 % and 11 %
         * faster measured). Only for heaps whose handle holds the same values
         * (matches()): the C++ Allocator picks it from its policies, the
         * library's kernels dispatch on matches(). */
        template<u32 RESET, u32 DIST, u32 OOM, u32 ALIGN>
        struct GpuIdsFixed : GpuIds
        {
            __device__ static __forceinline__ u32 reset(const mmc_device_handle&) { return RESET; }
            __device__ static __forceinline__ u32 distribution(const mmc_device_handle&) { return DIST; }
            __device__ static __forceinline__ u32 oom(const mmc_device_handle&) { return OOM; }
            __device__ static __forceinline__ u32 alignment(const mmc_device_handle&) { return ALIGN; }
            __host__ __device__ static bool matches(const mmc_device_handle& h)
            {
                return (h.resetfreedpages != 0u) == (RESET != 0u) && h.distribution == DIST && h.oom_policy == OOM
                       && (h.dataAlignment > 1u ? h.dataAlignment : 1u) == (ALIGN > 1u ? ALIGN : 1u);
            }
        };

        /* The configuration the bench's workloads and the reference's defaults
         * use: no page reset, XMallocSIMD, ReturnNull, Shrink<16>. */
        using GpuIdsDefault = GpuIdsFixed<0u, MMC_DIST_XMALLOCSIMD, MMC_OOM_RETURNNULL, 16u>;

        /* Base for a kernel whose requests never exceed a page after padding
         * (its caller knows the largest one): the multi-page search is left
         * out of it. That search is out-of-line code, and ptxas fits the
         * registers of every kernel that can call it around the search's own,
         * so a change in the search moved the chunk paths' register
         * allocation: the uniform stress kernel, which never asks for more
         * than 1 KiB, ran 2 to 17 % slower after changes to the search alone.
         * A request above a page in such a kernel returns NULL and sets
         * MMC_DEVERR_PAGEBASED. Frees are unchanged. */
        template<class Base>
        struct SmallRequests : Base
        {
            static constexpr bool pageBased = false;
        };

        /* The reference's CPU-backend semantics (mallocMC_utils.hpp:85-87, 99-101, 121-123, 134-136). */
        struct SerialIds
        {
            static constexpr u32 warpSize = 1u;
            static constexpr bool coalesce = false; /* XMallocSIMD.hpp:136-137 */
            static constexpr bool cachedHints = false;
            static constexpr bool pageBased = true;
            __device__ static __forceinline__ u32 laneid() { return 0u; }
            __device__ static __forceinline__ u32 warpid() { return 0u; }
            __device__ static __forceinline__ u32 smid() { return 0u; }
            __device__ static __forceinline__ u32 reset(const mmc_device_handle& h) { return h.resetfreedpages; }
            __device__ static __forceinline__ u32 distribution(const mmc_device_handle& h) { return h.distribution; }
            __device__ static __forceinline__ u32 oom(const mmc_device_handle& h) { return h.oom_policy; }
            __device__ static __forceinline__ u32 alignment(const mmc_device_handle& h) { return h.dataAlignment; }
        };

        /* ---------------------------------------------------- memory helpers */
        __device__ __forceinline__ u32 ld_rlx(const u32* p)
        {
            u32 v;
            asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
            return v;
        }
        __device__ __forceinline__ uint4 ld_rlx_v4(const u32* p)
        {
            uint4 v;
            asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                         : "l"(p)
                         : "memory");
            return v;
        }
        __device__ __forceinline__ void st_rlx(u32* p, u32 v)
        {
            asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
        }
        /* fence.release.gpu: this thread's earlier memory operations are
         * performed before its later writes and atomics, for every thread of
         * the GPU. (It measured 6 % faster on the uniform stress than
         * fence.acq_rel.gpu, which also orders the later reads; the free
         * needs only the release.) */
        __device__ __forceinline__ void release_fence() { asm volatile("fence.release.gpu;" ::: "memory"); }
        __device__ __forceinline__ u32 lanemask_lt()
        {
            u32 r;
            asm("mov.u32 %0, %%lanemask_lt;" : "=r"(r));
            return r;
        }
        /* The lanes that call malloc, free or available_slots together, read
         * once per call. Every warp-wide operation inside names this mask, or a
         * ballot over it taken before the branch its lanes take, so all the
         * lanes it names reach it. Reading the active lanes again inside a
         * branch is not sound here: with a reading in malloc, one in create and
         * one in the chunk claim, each made a value by a reduction over itself,
         * lanes left malloc ahead of the lane that allocates for them, and a
         * kernel without launch bounds got pointers put together from other
         * values (104 of 780 000 requests of 16 to 1024 bytes on 152 blocks). The
         * lanes of a user's loop meet here in different rounds of it. As a
         * volatile the mask is a value of its own for the compiler; that costs
         * 0 to 0.9 % on most workloads, and small batches of uneven jobs took 121
         * us so, 138 without. */
        __device__ __forceinline__ u32 calling_lanes()
        {
            volatile u32 lanes = __activemask();
            return lanes;
        }
        __device__ __forceinline__ u32 umin(u32 a, u32 b) { return a < b ? a : b; }
        __device__ __forceinline__ u32 umax(u32 a, u32 b) { return a > b ? a : b; }
        __device__ __forceinline__ u32 divup(u32 a, u32 b) { return (a + b - 1u) / b; }

        /* Shrink::applyPadding (Shrink.hpp:132-137) / Noop (alignmentPolicies/Noop.hpp:55-59). */
        __host__ __device__ __forceinline__ u32 apply_padding(u32 align, u32 bytes)
        {
            if(align <= 1u)
                return bytes;
            const u32 clear = align - 1u;
            return (bytes + clear) & ~clear;
        }

        __device__ __forceinline__ char* page_data(const mmc_device_handle& h, u32 page)
        {
            return h.pages + static_cast<u64>(page) * h.pagesize;
        }

        /* onPageMasksPosition, Scatter.hpp:315-318 */
        __device__ __forceinline__ u32* on_page_masks(const mmc_device_handle& h, u32 page, u32 nMasks)
        {
            return reinterpret_cast<u32*>(page_data(h, page) + h.pagesize - 4u * nMasks);
        }

        /* Page::init, Scatter.hpp:247-258: zero the words that can hold on-page masks. */
        __device__ __forceinline__ void page_init(const mmc_device_handle& h, u32 page)
        {
            u32* w = on_page_masks(h, page, h.maxOnPageMasks);
            for(u32 i = 0; i < h.maxOnPageMasks; ++i)
                st_rlx(w + i, 0u);
        }

        __device__ __forceinline__ void set_error(const mmc_device_handle& h, u32 bits)
        {
            atomicOr(&h.state->error_flags, bits);
        }

        /* ------------------------------------------------ free-page bitmap
         * h.freemap has one bit per page, set while the page's chunk size is
         * 0; the concurrent multi-page search reads it instead of the chunk
         * sizes, 32 pages per word (no counterpart in the reference, which
         * scans the page table). The chunk size stays the authority: a run is
         * owned only once markpages' CASes succeed, so a bit set on a used
         * page costs the search a failed CAS, as a lost run does. What must
         * not happen is a clear bit on a free page for longer than a free is
         * in flight, or the search would skip free pages. So: every change of
         * a chunk size to 0 (a free, a page reset, a markpages roll-back) sets
         * the bit after its CAS; every change from 0 clears the bit either
         * before its CAS, or after it while nothing can free the page yet
         * (markpages' run before it is handed out; a reset-mode format while
         * the caller holds a fill slot), and a fence then waits for the clear
         * to be performed, so no clear can land after a later free's set. */
        __device__ __forceinline__ void freemap_clear_acked(u32* fm, u32 page)
        {
            atomicAnd(&fm[page >> 5], ~(1u << (page & 31u)));
            asm volatile("fence.acq_rel.gpu;" ::: "memory");
        }

        __device__ __forceinline__ void freemap_set(u32* fm, u32 page)
        {
            atomicOr(&fm[page >> 5], 1u << (page & 31u));
        }

        /* Behind the free-page bitmap lies a second one, with the bits of the
         * pages that are in no multi-page run: all that a chunk walk has to
         * look at. A run clears its bits once it is marked (its asker's fence
         * waits for that before the run is handed out), and its free sets
         * them, with a fence, before the pages' chunk sizes go to 0: a bit may
         * stay set on a run's page, never clear on another. */
        __host__ __device__ __forceinline__ u32 freemap_words(u32 numpages) { return ((numpages / 32u + 4u) & ~3u) + 4u; }
        __device__ __forceinline__ u32* walkmap(u32* fm, u32 numpages) { return fm + freemap_words(numpages); }

        /* set (free) or clear the bits of pages [first, first + n), one atomic per word */
        __device__ inline void freemap_range(u32* fm, u32 first, u32 n, bool free)
        {
            for(u32 p = first, end = first + n; p < end;)
            {
                const u32 b = p & 31u;
                const u32 cnt = umin(32u - b, end - p);
                const u32 mask = cnt == 32u ? 0xFFFFFFFFu : ((1u << cnt) - 1u) << b;
                if(free)
                    atomicOr(&fm[p >> 5], mask);
                else
                    atomicAnd(&fm[p >> 5], ~mask);
                p += cnt;
            }
        }

        /* nextspot, Scatter.hpp:293-304 */
        __device__ __forceinline__ u32 nextspot(u32 bitfield, u32 spot, u32 spots)
        {
            const u32 low_part = (spot + 1u) == 32u ? 0u : (bitfield >> (spot + 1u));
            const u32 high_part = (bitfield << (spots - (spot + 1u)));
            const u32 selection_mask = spots == 32u ? ~0u : ((1u << spots) - 1u);
            bitfield = (high_part | low_part) & selection_mask;
            /* (spot + step) % spots; step is at most spots + 1 */
            u32 next = spot + static_cast<u32>(__ffs(static_cast<int>(~bitfield)));
            next -= next >= spots ? spots : 0u;
            return next - (next >= spots ? spots : 0u);
        }

        /* calcAdditionalChunks, Scatter.hpp:365-381: the (int) casts collapse to
         * unsigned arithmetic and CUDA's ::max/::min(int, unsigned) compare unsigned. */
        __device__ __forceinline__ u32 calc_additional_chunks(u32 pagesize, u32 fullsegments, u32 segmentsize,
                                                              u32 chunksize)
        {
            if(fullsegments != 32u)
                return umin(31u, (pagesize - fullsegments * segmentsize - 4u) / chunksize);
            return 0u;
        }

        /* Geometry of a page formatted with a chunk size (tryUsePage :493-508,
         * deallocChunked :652-660, countFreeChunksInPage :1116-1138). */
        struct ChunkGeom
        {
            bool hier;        /* chunksize <= HierarchyThreshold: on-page segment masks */
            u32 fullsegments; /* hierarchical: segments of 32 chunks */
            u32 additional;   /* hierarchical: chunks in the last, partial segment */
            u32 segments;     /* hierarchical: on-page mask words */
            u32 capacity;     /* chunks the page holds */
        };

        __device__ __forceinline__ ChunkGeom chunk_geom(const mmc_device_handle& h, u32 chunksize)
        {
            ChunkGeom g;
            g.hier = chunksize <= h.hierarchyThreshold;
            if(g.hier)
            {
                const u32 segmentsize = chunksize * 32u + 4u;
                g.fullsegments = umin(32u, h.pagesize / segmentsize);
                g.additional = calc_additional_chunks(h.pagesize, g.fullsegments, segmentsize, chunksize);
                g.segments = g.fullsegments + (g.additional > 0u ? 1u : 0u);
                g.capacity = g.fullsegments * 32u + g.additional;
            }
            else
            {
                g.fullsegments = g.additional = g.segments = 0u;
                g.capacity = umin(h.pagesize / chunksize, 32u);
            }
            return g;
        }

        /* Capacity of a page formatted with chunksize. */
        __device__ __forceinline__ u32 page_capacity(const mmc_device_handle& h, u32 chunksize)
        {
            return chunk_geom(h, chunksize).capacity;
        }

        /* n < page_capacity(h, chunksize), without its divisions: chunk n lies in
         * segment n / 32, which is a full one, or the last one and n % 32 below
         * its chunks (calc_additional_chunks, wrap and all). */
        __device__ __forceinline__ bool page_has_room(const mmc_device_handle& h, u32 chunksize, u32 n)
        {
            const u32 P = h.pagesize;
            if(chunksize > h.hierarchyThreshold)
                return n < 32u && (n + 1u) * chunksize <= P;
            const u32 segmentsize = 32u * chunksize + 4u;
            const u64 below = static_cast<u64>(n / 32u) * segmentsize; /* where its segment begins */
            const u32 spot = n % 32u;
            return n < 1024u
                && (below + segmentsize <= P
                    || (below <= P && spot < 31u && (spot + 1u) * chunksize <= P - static_cast<u32>(below) - 4u));
        }

        /* Claim one chunk on a page whose fill slot is reserved:
         * addChunkHierarchy (Scatter.hpp:397-421) for hierarchical pages,
         * addChunkNoHierarchy (:432-443) otherwise, both over usespot
         * (:329-347, first spot laneid % spots, randInit :277-281): atomicOr a
         * bit of a word (a segment's on-page mask or the page bitmask); when it
         * was set already, stop if the word is full, else try the next free
         * spot of the returned word. MMC_USESPOT_MAX_TRIES lost races count as
         * a full word, which every caller handles. `mask` is the page's
         * segment hints. One loop with one atomicOr serves both page kinds and
         * every retry: the copies of an unrolled retry loop in front of each
         * of them were most of a kernel's code (see alloc_chunked). */
        template<class Ids>
        __device__ __forceinline__ void* claim_chunk(const mmc_device_handle& h, u32 page, u32 chunksize,
                                                     const ChunkGeom& g, u32 mask)
        {
            u32* word = &h.bitmask[page];
            u32 spots = g.capacity;
            u32 seg = 0u;
            u32 tries = 1u;
            if(g.hier)
            {
                seg = Ids::laneid() % g.segments;
                if((mask & (1u << seg)) != 0u)
                    seg = nextspot(mask, seg, g.segments);
                tries = g.segments - static_cast<u32>(__popc(mask));
                word = on_page_masks(h, page, g.segments) + seg;
                spots = seg < g.fullsegments ? 32u : g.additional;
            }
            u32 spot = Ids::laneid() % spots;
            u32 races = 0u;
            bool claimed = false;
#pragma unroll 1
            while(!claimed && tries != 0u)
            {
                const u32 bit = 1u << spot;
                const u32 old = atomicOr(word, bit);
                claimed = (old & bit) == 0u;
                if(!claimed)
                {
                    if(static_cast<u32>(__popc(old)) < spots && ++races < MMC_USESPOT_MAX_TRIES)
                        spot = nextspot(old, spot, spots);
                    else if(--tries != 0u || g.hier)
                    {
                        atomicOr(&h.bitmask[page], 1u << seg);
                        /* A free in this segment may have cleared the hint just before
                         * it was set; undo a mark the segment no longer deserves so no
                         * stale "full" bit outlives the chunks. A lone thread only gets
                         * here for a full segment, so this never fires serially. */
                        if(static_cast<u32>(__popc(ld_rlx(word))) < spots)
                            atomicAnd(&h.bitmask[page], ~(1u << seg));
                        seg = nextspot(mask, seg, g.segments);
                        word = on_page_masks(h, page, g.segments) + seg;
                        spots = seg < g.fullsegments ? 32u : g.additional;
                        spot = Ids::laneid() % spots;
                        races = 0u;
                    }
                }
            }
            return claimed ? page_data(h, page) + (32u * seg + spot) * chunksize : nullptr;
        }

        /* tryUsePage, Scatter.hpp:454-518; [lo, hi] is isChunkSizeInRange (:586-588). */
        template<class Ids>
        __device__ __forceinline__ void* try_use_page(const mmc_device_handle& h, u32 page, u32 chunksize, u32 lo, u32 hi)
        {
            void* chunk_ptr = nullptr;
            /* the segment hints are read before the fill-count atomic so both
             * round trips overlap (the reference reads them just after it,
             * Scatter.hpp:404; alone on the heap both reads see the same word) */
            u32 mask = chunksize <= h.hierarchyThreshold ? ld_rlx(&h.bitmask[page]) : 0u;
            const u32 filllevel = atomicAdd(&h.count[page], 1u);
            const bool reset = Ids::reset(h) != 0u;
            bool tryAllocMem = !reset;
            if(reset && filllevel < h.pagesize)
            {
                const u32 oldChunksize = atomicCAS(&h.chunksize[page], 0u, chunksize);
                if(oldChunksize == 0u)
                    freemap_clear_acked(h.freemap, page); /* our fill slot keeps the page from a reset */
                if(oldChunksize == 0u || (oldChunksize >= lo && oldChunksize <= hi))
                    tryAllocMem = true;
                if(oldChunksize != 0u && oldChunksize != chunksize)
                {
                    chunksize = oldChunksize;
                    mask = ld_rlx(&h.bitmask[page]);
                }
            }
            if(tryAllocMem)
            {
                const ChunkGeom g = chunk_geom(h, chunksize);
                if(filllevel < g.capacity)
                    chunk_ptr = claim_chunk<Ids>(h, page, chunksize, g, mask);
            }
            if(chunk_ptr == nullptr)
                atomicSub(&h.count[page], 1u);
            return chunk_ptr;
        }

        /* One page of allocChunked's walk (Scatter.hpp:580-604), given the page's
         * chunk size as already loaded. The reference's CAS(0 -> minAllocation)
         * only writes a zero word; on a formatted page it just returns the value,
         * so it is issued only when the load saw zero. */
        template<class Ids>
        __device__ __forceinline__ void* attempt_page(const mmc_device_handle& h, u32 page, u32 before, u32 bytes,
                                                      u32 minAllocation, u32 maxchunksize)
        {
            if(before == 0u)
            {
                freemap_clear_acked(h.freemap, page);
                before = atomicCAS(&h.chunksize[page], 0u, minAllocation);
            }
            u32 use = 0u;
            if(before == 0u)
                use = minAllocation;
            else if(before >= bytes && before <= maxchunksize)
                use = before;
            if(use == 0u)
            {
                MMC_STAT(h, MMC_STAT_SIZE_MISMATCH);
                return nullptr;
            }
            void* r = try_use_page<Ids>(h, page, use, bytes, maxchunksize);
            if(r == nullptr)
                MMC_STAT(h, MMC_STAT_PAGE_FULL);
            return r;
        }

        /* The pages of one region a request may use, as two masks in page order
         * (bit i = page region_offset + i): unformatted pages (chunk size 0) and
         * pages formatted with a chunk size in [bytes, maxchunksize] that have
         * a chunk free. Every other page is one the reference's walk visits
         * only to find it formatted for another size, taken by a multi-page run
         * (Scatter.hpp:584-591) or full (:500). Chunk sizes, and where there
         * are chunk pages their fill counts, are read with 16-byte loads, 16 or
         * eight pages at once: a walk costs one round trip per region of
         * multi-page runs and three per region of full chunk pages, where
         * reserving a fill slot on each page and giving it back cost two per
         * page. (Keeping the chunk sizes of 16 pages for the second step takes
         * one round trip less and spilled 370 bytes of the stress kernel.)
         * `room`: the region has a page or a chunk of any size free. (With
         * pagesize / chunksize for what a page holds, which on-page masks make
         * too many for 16, 32 and 64 bytes in 4 KiB, regions of those never were
         * full and walks tried each of their pages: 1.8 M blocks of 64 bytes on
         * a 128 MiB heap, no distribution, 106 to 114 ms, now 11 to 12. The exact
         * test costs live data of 8 to 600 bytes 1.6 %, mixed sizes on a heap in
         * use 4 %.) Needs regionsize % 4 == 0 and regionsize <= 32. */
        __device__ __forceinline__ void region_candidates(const mmc_device_handle& h, u32 region_offset, u32 bytes,
                                                          u32 maxchunksize, u32& zero, u32& fit, bool& room)
        {
            const u32 R = h.regionsize;
            zero = 0u;
            fit = 0u;
            room = false;
            u32 chunks = 0u; /* pages formatted for chunks */
#pragma unroll 1
            for(u32 base = 0; base < R; base += 16u)
            {
                uint4 v[4];
#pragma unroll
                for(u32 k = 0; k < 4u; ++k)
                    v[k] = (base + 4u * k < R) ? ld_rlx_v4(&h.chunksize[region_offset + base + 4u * k])
                                               : make_uint4(~0u, ~0u, ~0u, ~0u);
#pragma unroll
                for(u32 k = 0; k < 4u; ++k)
                {
                    const u32 w[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
#pragma unroll
                    for(u32 j = 0; j < 4u; ++j)
                    {
                        zero |= (w[j] == 0u ? 1u : 0u) << ((base + 4u * k + j) & 31u);
                        chunks |= (w[j] - 1u < h.pagesize ? 1u : 0u) << ((base + 4u * k + j) & 31u);
                    }
                }
            }
#pragma unroll 1
            for(u32 base = 0; chunks >> base != 0u; base += 8u)
            {
                uint4 v[2], c[2];
#pragma unroll
                for(u32 k = 0; k < 2u; ++k)
                {
                    const bool in = base + 4u * k < R;
                    v[k] = in ? ld_rlx_v4(&h.chunksize[region_offset + base + 4u * k]) : make_uint4(~0u, ~0u, ~0u, ~0u);
                    c[k] = in ? ld_rlx_v4(&h.count[region_offset + base + 4u * k]) : make_uint4(0u, 0u, 0u, 0u);
                }
#pragma unroll
                for(u32 k = 0; k < 2u; ++k)
                {
                    const u32 w[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
                    const u32 n[4] = {c[k].x, c[k].y, c[k].z, c[k].w};
#pragma unroll
                    for(u32 j = 0; j < 4u; ++j)
                    {
                        const bool more = w[j] - 1u < h.pagesize && page_has_room(h, w[j], n[j]);
                        fit |= (w[j] >= bytes && w[j] <= maxchunksize && more ? 1u : 0u) << (base + 4u * k + j);
                        room = room || more;
                    }
                }
                if(base == 24u)
                    break;
            }
            room = room || zero != 0u;
        }

        /* allocChunked's two-pass region walk (Scatter.hpp:563-636), resumed
         * after the start page: in the first region of pass 0 the region
         * counter is the one already read (level) and the start page was tried.
         * The rest of that region is walked page by page, as the reference
         * walks it: most walks end there, after a page or two. Every further
         * region is read whole (region_candidates) and only its usable pages
         * are tried, in the reference's order from the entry page: a walk that
         * crosses regions of full pages or of multi-page runs costs a few
         * round trips per region instead of one or two per page. The region
         * counters are looked at eight regions ahead, so a stretch of regions
         * skipped as 3/4 full costs one round trip and one step per eight;
         * read with them, a word of the map of pages outside multi-page runs
         * has both passes skip the regions that runs fill as well. (The 32 GiB
         * fragmentation run's two waves up to its first NULL: 800 and 50 to
         * 1140 ms a region at a time, 850 and 915 by the counters alone, 226 and
         * 550 so; the whole run 2.2 to 3.4 s, now 1.3 s.) Alone on the heap every page gets
         * the reference's outcome, in the reference's order.
         *
         * The counters: the reference counts every failed walk, whatever size
         * it wanted, and passes regions that 3/4 * R have failed in. Many
         * threads raise them that far at once, in regions that still have room
         * for other sizes; walks then pass whole blocks with free chunks, the
         * first-free-block hint follows them, and new pages are formatted
         * further on. For concurrent callers a walk counts only in a region
         * with no page free and no chunk free of any size, and only in the
         * first pass (the second walks every region anyway, and would mark the
         * whole heap). The 32 GiB fragmentation run, whose multi-page requests
         * are served fast enough to fill the heap to its last page: 0.9713 of
         * the heap after its refill counting every walk, 0.978 this way (the
         * reference's serial run: 0.9750).
         *
         * One attempt serves every page, and malloc has one call of all this:
         * with an attempt for each kind of region, each with unrolled claim
         * retries, and two call sites in malloc, a kernel that allocates had
         * 100 to 180 KB of code, and instruction fetch was the first stall of
         * the stress and batched kernels.
         *
         * The lanes of a warp do not wait for one another in here: no step
         * names a mask, so a lane's walk ends by itself, after the pages of
         * 2 * numregions regions. (A form whose lanes stepped together, by a
         * vote over lanes read inside this branch, took 4.99 ms on the uniform
         * stress where this one takes 6.1, but a few launches in a hundred of a
         * 16 to 256 byte stress did not end. What masks read in branches did
         * elsewhere is at calling_lanes; the form was not run again.) */
        template<class Ids>
        __device__ __forceinline__ void* alloc_chunked_walk(const mmc_device_handle& h, u32 bytes, u32 minAllocation,
                                                            u32 maxchunksize, u32 start, u32 level)
        {
            const u32 R = h.regionsize;
            const u32 numregions = h.numregions;
            const bool batched = (R % 4u) == 0u && R <= 32u;
            const bool mapped = Ids::warpSize > 1u && batched && (R & (R - 1u)) == 0u; /* a region's bits lie in one word */
            const u32 rmask = R >= 32u ? 0xFFFFFFFFu : ((1u << R) - 1u);
            u32 region = start / R;
            const u32 s0 = start - region * R;
            u32 checklevel = R * 3u / 4u;
            u64 ahead = 0u; /* counters of the regions ahead, a byte each */
            u32 known = 1u; /* how many, with this one */
            u32 edge = 0u; /* the page where the next access block begins, once it is needed */
            u32 left = 2u * numregions; /* regions to visit, in both passes, this one included */
            /* Visiting index i is page region * R + (s0 + i) % R. With masks, the
             * usable pages (todo) and the unformatted ones (zero) go by it;
             * without, i is the last page visited. */
            u32 todo = 0u, zero = 0u, i = 0u;
            bool masks = false;
            bool room = true; /* the region has a page or a chunk of some size free */
            bool walking = level < checklevel;
            if(!walking)
                i = R;
            void* res = nullptr;
            bool go = true;
            do
            {
                bool read = false;
                if(Ids::warpSize > 1u && go && walking && batched && !masks && i + 1u >= R)
                    read = true; /* walked page by page: is it full? */
                else if(go && (masks ? todo == 0u : i + 1u >= R))
                {
                    /* the region has no page left to try: on to the next one to walk */
                    if(walking && (Ids::warpSize == 1u || !batched || !room))
                    {
                        if(level + 1u <= R && (Ids::warpSize == 1u || checklevel <= R))
                            atomicCAS(&h.regions[region], level, level + 1u);
                        MMC_STAT(h, MMC_STAT_REGION_FAIL);
                    }
                    else
                        MMC_STAT(h, MMC_STAT_REGION_SKIP);
                    if(edge == 0u)
                        edge = (region * R / h.pagesperblock + 1u) * h.pagesperblock;
                    /* with it, the regions behind it that are passed by their
                     * counters, as far as those are known, up to the pass's end */
                    u32 n = 1u;
                    if(Ids::warpSize > 1u && checklevel <= 255u)
                    {
                        const u32 check = checklevel * 0x01010101u;
                        const u64 rest = ahead >> 8;
                        const u32 lo = ~__vcmpgeu4(static_cast<u32>(rest), check);
                        const u32 hi = ~__vcmpgeu4(static_cast<u32>(rest >> 32), check);
                        const u32 full = static_cast<u32>(lo != 0u ? __ffs(static_cast<int>(lo)) - 1
                                                                    : 32 + ((__ffs(static_cast<int>(hi)) - 1) & 31)) / 8u;
                        n += umin(umin(full, known - 1u), (left > numregions ? left - numregions : left) - 1u);
                    }
                    region += n;
                    if(region == numregions)
                        region = 0u;
                    if(region * R >= edge || region == 0u)
                    {
                        /* racy by design (Scatter.hpp:625-628) */
                        const u32 access_block_id = region * R / h.pagesperblock;
                        if(s0 == 0u && (region * R == access_block_id * h.pagesperblock || h.pagesperblock % R == 0u)
                           && access_block_id > ld_rlx(&h.state->firstfreeblock))
                            st_rlx(&h.state->firstfreeblock, access_block_id);
                        edge = (access_block_id + 1u) * h.pagesperblock;
                    }
                    ahead = n < 8u ? ahead >> (8u * n) : 0u;
                    known -= n;
                    left -= n;
                    if(left == numregions)
                    {
                        /* the second pass walks every region */
                        checklevel = R + 1u;
                        known = 0u;
                    }
                    go = left != 0u;
                    if(known == 0u && go)
                    {
                        known = umin(8u, numregions - region);
                        ahead = 0u;
#pragma unroll
                        for(u32 k = 0; k < 8u; ++k)
                            if(k < known)
                            {
                                u32 full = umin(ld_rlx(&h.regions[region + k]), 255u);
                                if(mapped)
                                {
                                    const u32 first = (region + k) * R;
                                    const u32 look = ld_rlx(&walkmap(h.freemap, h.numpages)[first >> 5]) >> (first & 31u);
                                    full = (look & rmask) != 0u ? full : 255u;
                                }
                                ahead |= static_cast<u64>(full) << (8u * k);
                            }
                    }
                    /* the counter as it was looked at, up to eight regions ago: of
                     * several walks that fail here together one raises it */
                    level = static_cast<u32>(ahead) & 255u;
                    /* of large regions a byte does not hold the counter that decides */
                    if(go && level == 255u && checklevel > 255u)
                        level = ld_rlx(&h.regions[region]);
                    walking = go && level < checklevel;
                    masks = batched;
                    todo = 0u;
                    i = walking ? ~0u : R;
                    read = walking && batched;
                }
                if(read)
                {
                    region_candidates(h, region * R, bytes, maxchunksize, zero, todo, room);
                    if(s0 != 0u)
                    {
                        zero = ((zero >> s0) | (zero << (R - s0))) & rmask;
                        todo = ((todo >> s0) | (todo << (R - s0))) & rmask;
                    }
                    todo = masks ? todo | zero : 0u;
                    masks = true;
                }
                if(go && (masks ? todo != 0u : i + 1u < R))
                {
                    ++i;
                    if(masks)
                    {
                        i = static_cast<u32>(__ffs(static_cast<int>(todo))) - 1u;
                        todo &= todo - 1u;
                    }
                    const u32 off = s0 + i;
                    const u32 page = region * R + (off >= R ? off - R : off);
                    MMC_STAT(h, MMC_STAT_WALK_PAGES);
                    const u32 before = masks && ((zero >> i) & 1u) != 0u ? 0u : ld_rlx(&h.chunksize[page]);
                    res = attempt_page<Ids>(h, page, before, bytes, minAllocation, maxchunksize);
                    go = res == nullptr;
                }
                /* (keeps the compiler from threading the next step's jumps) */
                asm volatile("" ::: "memory");
            } while(go);
            return res;
        }

        /* One page of a same-size group claim, by the group's leader: reserve up
         * to `want` fill slots with one atomicAdd (the reference's per-chunk
         * check, filllevel < capacity, applied to k reservations at once), claim
         * as many free bits of the page's bitmask with atomicOr, give back what
         * found no bit. Pages of chunks above HierarchyThreshold only (their
         * bitmask maps chunks directly). Returns the claimed bits. */
        __device__ __forceinline__ u32 claim_bits_on_page(const mmc_device_handle& h, u32 page, u32 use, u32 want)
        {
            const u32 cap = umin(h.pagesize / use, 32u);
            const u32 old = atomicAdd(&h.count[page], want);
            u32 grant = old < cap ? umin(want, cap - old) : 0u;
            if(grant < want)
                atomicSub(&h.count[page], want - grant);
            const u32 full = cap == 32u ? 0xFFFFFFFFu : ((1u << cap) - 1u);
            u32 mask = grant != 0u ? ld_rlx(&h.bitmask[page]) : full;
            u32 got = 0u;
#pragma unroll 1
            for(u32 tries = 0; grant != 0u && tries < MMC_USESPOT_MAX_TRIES; ++tries)
            {
                u32 free = ~mask & full;
                if(free == 0u)
                    break;
                u32 pick = 0u;
#pragma unroll 1
                for(u32 n = 0; n < grant && free != 0u; ++n)
                {
                    pick |= free & (0u - free); /* lowest free bit */
                    free &= free - 1u;
                }
                const u32 prev = atomicOr(&h.bitmask[page], pick);
                const u32 mine = pick & ~prev;
                got |= mine;
                grant -= static_cast<u32>(__popc(mine));
                mask = prev | pick;
            }
            if(grant != 0u)
                atomicSub(&h.count[page], grant); /* reserved slots no bit was found for */
            return got;
        }

        /* Same-size claims: lanes of a warp asking for the same size hash to the
         * same first page (the hash depends on the size, the SM and the warp,
         * not the lane), where the reference has each of them reserve a fill
         * slot and claim a bit on its own, all contending for one count word and
         * one bitmask word. Here the lanes are grouped by size (the whole warp
         * when a min/max reduction shows one size, else __match_any_sync, groups
         * of four lanes or more), and the group's lowest lane claims for all of
         * them, page by page through the first region in the walk's order
         * (claim_bits_on_page); the lane of rank r takes the r-th chunk claimed.
         * Lanes left over go the usual way. Measured on GB300: a warp-uniform
         * 256 B / 512 B / 1 KiB stress runs 1.7x / 2.9x / 2.4x faster, the
         * mixed-size stress 2.6 % faster (smaller groups cost more than they
         * save, hence the four-lane floor). `am`: the lanes that come here, all
         * of them. Returns true with `out` set when this lane got its chunk. */
        template<class Ids>
        __device__ __forceinline__ bool claim_same_size(const mmc_device_handle& h, u32 am, u32 bytes, u32 minAllocation,
                                                        u32 maxchunksize, u32 start, u32 fill0, u32 cs0, void*& out)
        {
            if(Ids::reset(h))
                return false;
            const bool same = __reduce_min_sync(am, bytes) == __reduce_max_sync(am, bytes);
            const u32 peers = same ? am : __match_any_sync(am, bytes);
            const u32 k = static_cast<u32>(__popc(peers));
            /* sizes whose pages could be hierarchical keep the one-lane claim */
            if(k < 4u || minAllocation <= h.hierarchyThreshold)
                return false;
            const u32 lane = Ids::laneid();
            const int leader = __ffs(static_cast<int>(peers)) - 1;
            const bool lead = lane == static_cast<u32>(leader);
            const u32 rank = static_cast<u32>(__popc(peers & lanemask_lt()));
            const u32 R = h.regionsize;
            const u32 region_ok = __shfl_sync(peers, fill0 < R * 3u / 4u ? 1u : 0u, leader);
            if(region_ok == 0u)
                return false;
            /* the leader's start page: the others' may be another, where they
             * read the first-free-block hint apart and it moved in between */
            u32 page = __shfl_sync(peers, start, leader);
            const u32 region_offset = (page / R) * R;
            u32 served = 0u;
#pragma unroll 1
            for(u32 visited = 0; visited < R && served < k; ++visited)
            {
                u32 got = 0u, use = 0u;
                if(lead)
                {
                    u32 before = visited == 0u ? cs0 : ld_rlx(&h.chunksize[page]);
                    if(before == 0u)
                    {
                        freemap_clear_acked(h.freemap, page);
                        before = atomicCAS(&h.chunksize[page], 0u, minAllocation);
                    }
                    use = before == 0u ? minAllocation : ((before >= bytes && before <= maxchunksize) ? before : 0u);
                    if(use > h.hierarchyThreshold)
                        got = claim_bits_on_page(h, page, use, k - served);
                }
                got = __shfl_sync(peers, got, leader);
                use = __shfl_sync(peers, use, leader);
                const u32 n = static_cast<u32>(__popc(got));
                if(rank >= served && rank < served + n)
                {
                    u32 m = got;
#pragma unroll 1
                    for(u32 i = served; i < rank; ++i)
                        m &= m - 1u;
                    const u32 bit = static_cast<u32>(__ffs(static_cast<int>(m))) - 1u;
                    out = page_data(h, page) + bit * use;
                }
                served += n;
                page = region_offset + ((page + 1u) % R);
            }
            if(rank < served)
            {
                MMC_STAT(h, MMC_STAT_FIRST_PAGE);
                return true;
            }
            return false;
        }

        /* allocChunked, Scatter.hpp:527-637. The walk's first page is tried with
         * its region counter and chunk size read together, as straight-line
         * code every lane of a warp executes in step; only lanes whose first
         * page fails enter the (divergent) rest of the walk. `lanes`: the
         * lanes that call this together. */
        template<class Ids>
        __device__ __forceinline__ void* alloc_chunked(const mmc_device_handle& h, u32 lanes, u32 bytes)
        {
            const u32 P = h.pagesize;
            const u32 R = h.regionsize;
            const u32 minAllocation = umax(bytes, h.paddedMinChunkSize);
            const u32 numpages = h.numpages;
            const u32 pagesperblock = h.pagesperblock;
            const u32 reloff = Ids::warpSize * minAllocation / P;
            const u32 start_page_in_block = (minAllocation * h.hashingK + h.hashingDistMP * Ids::smid()
                                             + (h.hashingDistWP + h.hashingDistWPRel * reloff) * Ids::warpid())
                % pagesperblock;
            const u32 maxchunksize = umin(P, umax(h.wastefactor * bytes, h.paddedMinChunkSize));
            const u32 ffb = Ids::cachedHints ? __ldca(&h.state->firstfreeblock) : ld_rlx(&h.state->firstfreeblock);
            u32 global_start_page = start_page_in_block + ffb * pagesperblock;
            if(global_start_page >= numpages)
                global_start_page %= numpages; /* unreachable for a consistent header; keeps accesses in bounds */

            const u32 fill0 = ld_rlx(&h.regions[global_start_page / R]);
            const u32 cs0 = ld_rlx(&h.chunksize[global_start_page]);
            MMC_STAT(h, MMC_STAT_CHUNKED);
            void* res = nullptr;
            bool served = false;
            if constexpr(Ids::warpSize > 1u)
            {
                served = claim_same_size<Ids>(h, lanes, bytes, minAllocation, maxchunksize, global_start_page, fill0, cs0,
                                              res);
            }
            if(!served && fill0 < R * 3u / 4u)
            {
                res = attempt_page<Ids>(h, global_start_page, cs0, bytes, minAllocation, maxchunksize);
                if(res != nullptr)
                    MMC_STAT(h, MMC_STAT_FIRST_PAGE);
            }
            if(res == nullptr)
            {
                res = alloc_chunked_walk<Ids>(h, bytes, minAllocation, maxchunksize, global_start_page, fill0);
                if(res == nullptr)
                    MMC_STAT(h, MMC_STAT_CHUNKED_FAIL);
            }
            return res;
        }

        /* deallocChunked, Scatter.hpp:646-736 */
        template<class Ids>
        __device__ void dealloc_chunked(const mmc_device_handle& h, void* mem, u32 page, u32 chunksize)
        {
            const u32 P = h.pagesize;
            const u32 inpage_offset = static_cast<u32>(static_cast<char*>(mem) - page_data(h, page));
            u32 segment;
            if(chunksize <= h.hierarchyThreshold)
            {
                const ChunkGeom g = chunk_geom(h, chunksize);
                segment = inpage_offset / (chunksize * 32u);
                const u32 withinsegment = (inpage_offset - segment * (chunksize * 32u)) / chunksize;
                atomicAnd(on_page_masks(h, page, g.segments) + segment, ~(1u << withinsegment));
            }
            else
                segment = inpage_offset / chunksize;
            /* both kinds clear their bit of the page bitmask (:665, :670) */
            atomicAnd(&h.bitmask[page], ~(1u << segment));

            u32 oldfilllevel = 0u;
            if(Ids::reset(h))
            {
                oldfilllevel = atomicCAS(&h.count[page], 1u, P);
                bool locked = oldfilllevel == 1u;
                if(!locked)
                {
                    oldfilllevel = atomicSub(&h.count[page], 1u);
                    /* The reference resets a page only when a freer's CAS sees
                     * count == 1, so two last frees racing past each other leave
                     * it formatted. A freer that took the count from 1 to 0 takes
                     * the same lock (count = pagesize) if nobody has claimed the
                     * page since; a lone thread never gets here with old == 1. */
                    if(oldfilllevel == 1u)
                        locked = atomicCAS(&h.count[page], 0u, P) == 0u;
                }
                if(locked)
                {
                    page_init(h, page);
                    /* no chunk is live under the lock: drop any segment hint a
                     * race left behind (a no-op for the reference's serial runs) */
                    atomicExch(&h.bitmask[page], 0u);
                    if(atomicCAS(&h.chunksize[page], chunksize, 0u) == chunksize)
                        freemap_set(h.freemap, page);
                    __threadfence();
                    atomicSub(&h.count[page], P);
                }
            }
            else
                oldfilllevel = atomicSub(&h.count[page], 1u);

            if(oldfilllevel == P / 2u / chunksize)
            {
                const u32 region = page / h.regionsize;
                atomicExch(&h.regions[region], 0u);
                const u32 block = page / h.pagesperblock;
                if(Ids::warpid() + Ids::laneid() == 0u)
                    atomicMin(&h.state->firstfreeblock, block);
            }
        }

        /* chunk size seen by the page-based scan; index numpages (one past the end,
         * which the reference's second search reads) counts as "in use". */
        __device__ __forceinline__ u32 scan_chunksize(const mmc_device_handle& h, u32 page)
        {
            return page < h.numpages ? ld_rlx(&h.chunksize[page]) : 1u;
        }

        /* markpages, Scatter.hpp:745-764 (the serial form): CAS(chunksize,
         * 0 -> bytes) page by page; on a failure the pages already set are put
         * back with CAS(bytes -> 0). */
        __device__ inline bool markpages(const mmc_device_handle& h, u32 startpage, u32 pages, u32 bytes)
        {
            u32 abord = 0xFFFFFFFFu;
            for(u32 trypage = startpage; trypage < startpage + pages; ++trypage)
            {
                const u32 old = atomicCAS(&h.chunksize[trypage], 0u, bytes);
                if(old != 0u)
                {
                    abord = trypage;
                    break;
                }
            }
            if(abord == 0xFFFFFFFFu)
            {
                freemap_range(h.freemap, startpage, pages, false);
                asm volatile("fence.acq_rel.gpu;" ::: "memory");
                return true;
            }
            for(u32 trypage = startpage; trypage < abord; ++trypage)
                if(atomicCAS(&h.chunksize[trypage], bytes, 0u) == bytes)
                    freemap_set(h.freemap, trypage);
            return false;
        }

        /* allocPageBasedSingleRegion, Scatter.hpp:775-813 */
        __device__ inline void* alloc_page_based_single_region(const mmc_device_handle& h, u32 startpage, u32 endpage,
                                                        u32 bytes)
        {
            const u32 pagestoalloc = divup(bytes, h.pagesize);
            u32 freecount = 0;
            bool left_free = false;
            for(u32 search_page = startpage + 1u; search_page > endpage;)
            {
                --search_page;
                if(scan_chunksize(h, search_page) == 0u)
                {
                    if(++freecount == pagestoalloc)
                    {
                        if(search_page + pagestoalloc <= h.numpages && markpages(h, search_page, pagestoalloc, bytes))
                        {
                            if(!left_free)
                            {
                                /* the reference stores search_page - 1, which wraps for a
                                 * run ending at page 0 (Scatter.hpp:800-804) */
                                u32 nf = search_page - 1u;
                                if(!h.reference_quirks && search_page == 0u)
                                    nf = 0u;
                                atomicCAS(&h.state->firstFreePageBased, startpage, nf);
                            }
                            return page_data(h, search_page);
                        }
                    }
                }
                else
                {
                    left_free = true;
                    freecount = 0;
                }
            }
            return nullptr;
        }

        /* allocPageBasedSingle, Scatter.hpp:824-840, with a bounded, backed-off
         * mutex wait: the reference's serial protocol, used for SerialIds. */
        __device__ inline void* alloc_page_based_single(const mmc_device_handle& h, u32 bytes)
        {
            u32 ns = 32u;
            for(u32 it = 0; atomicExch(&h.state->pagebasedMutex, 1u) != 0u; ++it)
            {
                if(it >= MMC_MUTEX_MAX_SPINS)
                {
                    set_error(h, MMC_DEVERR_TIMEOUT);
                    return nullptr;
                }
                __nanosleep(ns);
                if(ns < 2048u)
                    ns <<= 1;
            }
            __threadfence();
            const u32 spage = ld_rlx(&h.state->firstFreePageBased);
            void* res = alloc_page_based_single_region(h, spage, 0u, bytes);
            if(res == nullptr)
                res = alloc_page_based_single_region(h, h.numpages, spage, bytes);
            __threadfence();
            atomicExch(&h.state->pagebasedMutex, 0u);
            return res;
        }

        /* What the concurrent page-based search needs of the handle. */
        struct PageScan
        {
            u32* chunksize;
            u32* freemap;
            mmc_heap_state* state;
            char* pages;
            u32 numpages;
            u32 pagesize;
            u32 reference_quirks;
        };

        /* markpages (Scatter.hpp:745-764) for concurrent callers. The run's
         * top page is claimed first, alone: searches that meet one free
         * stretch all settle on runs ending at its top page, and that CAS lets
         * exactly one of them go on, while the others lose it holding no page
         * (a claim that lost part way would put back pages that concurrent
         * searches saw taken and settled below, leaving a hole of a page or
         * two that no multi-page run fits). The other pages' CASes go out 4 at
         * a time (independent atomics in flight together, not one round trip
         * per page); on a failure every page this call set is put back with
         * CAS(bytes -> 0), as the reference's roll-back does, and gets its
         * free-page bit back. A run that is marked has its bits cleared (and
         * the clears performed) before it is handed out. With no concurrent
         * caller the outcome is the serial form's, which claims upward. */
        __device__ __forceinline__ bool markpages_batched(const PageScan& c, u32 startpage, u32 pages, u32 bytes,
                                                          u32& free_below, u32& top_owner)
        {
            const u32 end = startpage + pages;
            top_owner = atomicCAS(&c.chunksize[end - 1u], 0u, bytes);
            if(top_owner != 0u)
            {
                /* the pages below the top were free in the search */
                free_below = pages - 1u;
                return false;
            }
            const u32 last = end - 1u;
            for(u32 base = startpage; base < last; base += 4u)
            {
                u32 old[4];
#pragma unroll
                for(u32 k = 0; k < 4u; ++k)
                    old[k] = (base + k < last) ? atomicCAS(&c.chunksize[base + k], 0u, bytes) : 0u;
                u32 lost = 0u;
#pragma unroll
                for(u32 k = 0; k < 4u; ++k)
                    lost |= (old[k] != 0u ? 1u : 0u) << k;
                if(lost != 0u)
                {
                    u32 top_back = 0u; /* highest page put back, plus one */
                    if(atomicCAS(&c.chunksize[last], bytes, 0u) == bytes)
                    {
                        freemap_set(c.freemap, last);
                        top_back = end;
                    }
                    for(u32 trypage = startpage; trypage < base; ++trypage)
                        if(atomicCAS(&c.chunksize[trypage], bytes, 0u) == bytes)
                        {
                            freemap_set(c.freemap, trypage);
                            top_back = umax(top_back, trypage + 1u);
                        }
#pragma unroll
                    for(u32 k = 0; k < 4u; ++k)
                        if(base + k < last && ((lost >> k) & 1u) == 0u
                           && atomicCAS(&c.chunksize[base + k], bytes, 0u) == bytes)
                        {
                            freemap_set(c.freemap, base + k);
                            top_back = umax(top_back, base + k + 1u);
                        }
                    /* Pages put back are freed pages, and a free raises the
                     * search hint over them (deallocPageBased's atomicMax,
                     * Scatter.hpp:885): while this claim held them, concurrent
                     * searches saw them used and may have settled below them
                     * and lowered the hint, which would leave them a hole no
                     * later search visits. */
                    if(top_back != 0u)
                        atomicMax(&c.state->firstFreePageBased, top_back - 1u);
                    /* the pages from startpage up to the lowest lost one were free */
                    free_below = base + static_cast<u32>(__ffs(static_cast<int>(lost))) - 1u - startpage;
                    return false;
                }
            }
            freemap_range(c.freemap, startpage, pages, false);
            freemap_range(walkmap(c.freemap, c.numpages), startpage, pages, false);
            asm volatile("fence.acq_rel.gpu;" ::: "memory");
            return true;
        }

        constexpr u32 kNoRun = 0xFFFFFFFFu;
        /* lost runs a concurrent multi-page search looks at again before it
         * settles below them */
        constexpr u32 kLostRunRetries = 8u;

        /* Bits b_hi down to b_lo of free-page word w (value x), continuing a
         * downward count of consecutive free pages: returns the first page of
         * a run of n free pages once the count reaches n, else kNoRun. A used
         * page resets the count; one that ends a stretch of two or more free
         * pages the search could not use marks those pages as left behind
         * (left_free), which keeps the search from lowering the hint past
         * them. A single free page between used ones is not counted: no
         * multi-page run (two pages at least) can use it until a neighbour is
         * freed, and that free raises the hint again. (The
         * reference marks every used page, so its hint also stays above
         * stretches of used pages it passed. Lowering it past those spares
         * every later search the rescan and moves no placement while the pages
         * stay used; a run freed there raises the hint again. Only a chunk
         * page reset to free there under resetfreedpages, which raises no
         * hint, is then found by the search from the top instead.) */
        __device__ __forceinline__ u32 scan_freemap_word(u32 x, u32 w, u32 b_hi, u32 b_lo, u32 n, u32& freecount,
                                                         bool& left_free)
        {
            const u32 span = b_hi - b_lo + 1u;
            const u32 mask = span == 32u ? 0xFFFFFFFFu : ((1u << span) - 1u) << b_lo;
            const u32 xm = x & mask;
            if(xm == mask)
            {
                if(freecount + span >= n)
                    return 32u * w + b_hi - (n - freecount - 1u);
                freecount += span;
                return kNoRun;
            }
            if(xm == 0u)
            {
                left_free = left_free || freecount > 1u;
                freecount = 0u;
                return kNoRun;
            }
            for(u32 b = b_hi + 1u; b-- > b_lo;)
            {
                if((xm >> b) & 1u)
                {
                    if(++freecount == n)
                        return 32u * w + b;
                }
                else
                {
                    left_free = left_free || freecount > 1u;
                    freecount = 0u;
                }
            }
            return kNoRun;
        }

        /* allocPageBasedSingleRegion's search (Scatter.hpp:775-813) for concurrent
         * callers, without the global mutex. It visits the pages the reference
         * visits, startpage down to endpage, and counts free runs as the
         * reference counts them (downward, reset at a used page), but reads the
         * free-page bitmap: 16 words, 512 pages, per round trip, with whole
         * words of free or used pages taken in one step. markpages' CAS on the
         * chunk sizes decides who owns a run, top page first. A lane that
         * loses the top page learns the winner's size from the CAS and goes on
         * right below the winner's run (every search that met the same free
         * stretch settled on a run ending at its top page), from the bitmap
         * words it has already read: the lanes that meet one stretch together
         * pack their runs into it one below the other, with no page left
         * between them, as the reference's serial search would. A lane that
         * loses a page below the top (a claim that settled elsewhere) looks
         * at the run again a few times, since that claim may be put back,
         * then keeps counting below the lost page. The hint is lowered as the
         * reference lowers it, to just below the run by a CAS from the value
         * the search started at, when the search left no free page behind.
         * With no concurrent caller this finds the reference's run. */
        __device__ __forceinline__ char* alloc_page_based_scan(const PageScan& c, u32 startpage, u32 endpage,
                                                               u32 bytes)
        {
            const u32 n = divup(bytes, c.pagesize);
            u32 freecount = 0u;
            bool left_free = false;
            u32 retries = 0u;
            const u32 wend = endpage >> 5;
            /* pages top-1, top-2, ..., endpage remain (top wraps to 0 for the
             * reference's underflowed hint: then nothing is visited); a start
             * past page numpages, which no consistent hint holds, is cut to it
             * so every bitmap word read lies inside the map */
            if(startpage > c.numpages && startpage != 0xFFFFFFFFu)
                startpage = c.numpages;
            u32 top = startpage + 1u;
            u32 g0 = 0u;
            uint4 grp[4];
            bool reuse = false; /* the window read last still holds word whi */
            while(top > endpage)
            {
                const u32 whi = (top - 1u) >> 5;
                if(!(reuse && whi <= g0 + 3u && whi + 12u >= g0))
                {
                    g0 = whi & ~3u; /* 16-byte group holding word whi */
#pragma unroll
                    for(u32 k = 0; k < 4u; ++k)
                        grp[k] = (g0 >= 4u * k && g0 - 4u * k + 3u >= wend)
                                     ? __ldcg(reinterpret_cast<const uint4*>(c.freemap + (g0 - 4u * k)))
                                     : make_uint4(0u, 0u, 0u, 0u);
                }
                reuse = false;
                u32 q = kNoRun;
                u32 wl = whi; /* lowest word scanned */
                /* Not unrolled: ptxas fits the registers of every kernel that
                 * calls malloc around this out-of-line search's own, and the
                 * unrolled loop (the window held in registers) made the
                 * uniform stress kernel spill and run 17 % slower. */
#pragma unroll 1
                for(u32 j = 0; j < 16u; ++j)
                {
                    if(g0 + 3u < j)
                        break; /* below word 0 */
                    const u32 w = g0 + 3u - j;
                    if(w > whi)
                        continue;
                    if(w < wend)
                        break;
                    const uint4 G = grp[j / 4u];
                    const u32 comp = 3u - (j % 4u);
                    const u32 x = comp == 3u ? G.w : (comp == 2u ? G.z : (comp == 1u ? G.y : G.x));
                    wl = w;
                    if(x == 0u)
                        MMC_STAT(c, MMC_STAT_PAGE_SCAN_USED);
                    q = scan_freemap_word(x, w, w == whi ? ((top - 1u) & 31u) : 31u, w == wend ? (endpage & 31u) : 0u,
                                          n, freecount, left_free);
                    if(q != kNoRun)
                        break;
                }
                MMC_STAT_ADD(c, MMC_STAT_PAGE_SCAN, 32u * (whi - wl + 1u));
                if(q == kNoRun)
                {
                    top = wl == wend ? endpage : 32u * wl;
                    continue;
                }
                u32 free_below = 0u, top_owner = 0u;
                if(q + n <= c.numpages && markpages_batched(c, q, n, bytes, free_below, top_owner))
                {
                    if(!left_free)
                    {
                        /* the reference stores q - 1, which wraps for a run
                         * ending at page 0 (Scatter.hpp:800-804) and leaves
                         * every later search empty; fixed mode stores 0 */
                        const u32 nf = (!c.reference_quirks && q == 0u) ? 0u : q - 1u;
                        atomicCAS(&c.state->firstFreePageBased, startpage, nf);
                    }
                    return c.pages + static_cast<u64>(q) * c.pagesize;
                }
                MMC_STAT(c, MMC_STAT_PAGE_LOST);
                if(top_owner != 0u)
                {
                    /* The run's top page went to a concurrent claim: a chunk
                     * page, or a run of top_owner bytes, which in the common
                     * case ends at that page (the searches that meet one free
                     * stretch settle on runs ending at its top). Go on below
                     * it, without waiting for its claim to show in the map. */
                    const u32 skip = top_owner > c.pagesize ? divup(top_owner, c.pagesize) : 1u;
                    const u32 qt = q + n; /* lost top page, plus one */
                    top = qt > skip ? qt - skip : 0u;
                    freecount = 0u;
                    reuse = true;
                    continue;
                }
                if(retries < kLostRunRetries)
                {
                    /* Look at the run's pages again, after a short backoff:
                     * the claim that beat this one may itself lose elsewhere
                     * and put its pages back, and two searches that take each
                     * other's pages both lose. Going on below the lost page at
                     * once would leave the top of the contested stretch to a
                     * later search that may never come (a hole of a page or
                     * two among the runs); the page above the run is used (or
                     * above the start), so counting restarts from 0 there. */
                    __nanosleep(64u << umin(retries, 4u));
                    ++retries;
                    top = q + n;
                    freecount = 0u;
                    continue;
                }
                /* the run below the lost page is still free: keep counting it,
                 * from the page below q */
                freecount = free_below;
                left_free = true;
                top = q;
            }
            return nullptr;
        }

        /* allocPageBased, Scatter.hpp:848-866, for concurrent callers: every
         * lane searches at once, lock-free (alloc_page_based_scan), where the
         * reference's mutex serialises every large request of the GPU and each
         * search walks the page table one round trip per page. Out of line (with
         * its context by value): kept out of every kernel body that calls malloc,
         * the multi-page code no longer crowds the instruction cache of the
         * chunk path; that measured 12 % faster on the uniform stress. */
        __device__ __noinline__ inline char* alloc_page_based_concurrent(const PageScan c, u32 bytes)
        {
            const u32 spage = ld_rlx(&c.state->firstFreePageBased);
            char* res = alloc_page_based_scan(c, spage, 0u, bytes);
            if(res == nullptr)
                res = alloc_page_based_scan(c, c.numpages, spage, bytes);
            if(res == nullptr)
                MMC_STAT(c, MMC_STAT_PAGE_BASED_FAIL);
            return res;
        }

        /* ---------------------------- multi-page requests of whole warps
         * Every concurrent search of the lock-free form above settles on the
         * same run, the topmost that fits, and one of them gets it per round
         * trip while all the others CAS the same word: a wave of 77 824
         * requests on an 8 GiB heap, 7 800 of them multi-page, took 19 to
         * 28 ms and 46 to 60 M atomics. (Served as below: 7 680 multi-page
         * requests on an empty 8 GiB heap 55 -> 0.4 ms, among half a heap of
         * freed and live runs 98 -> 9 ms.) Here a warp whose 32 lanes call malloc
         * together puts its lanes' requests in a ring, and whichever waiting
         * warp finds the lock free serves all that wait, up to 256 at a time:
         *   - it takes the topmost free stretch at the hint for the whole
         *     batch with one read of its bitmap words, when it is long enough;
         *   - else it streams the bitmap down from the hint once per batch,
         *     1024 pages at a time (a word per lane, four such windows in
         *     flight), and gives each window's topmost run that fits to the
         *     largest request it fits, until the window takes no more.
         * Either is some serial order of the batch's first-fit searches, so
         * the packing is the serial search's. The server clears the runs'
         * bits; each asking warp then marks its own runs' chunk sizes, 32
         * pages per instruction. Those CASes stay the authority: a run that
         * a chunk page took a page of is put back and asked for again.
         * Partial warps and requests above kServiceMaxPages keep the
         * lock-free search. */
        constexpr u32 kPageAsk = 0x80000000u; /* ring word of a waiting request */
        constexpr u32 kPageGone = 0xC0000000u; /* ring word of a request given up: | pages */
        constexpr u32 kPageAnswer = 0x40000000u; /* ring word of an answer: | first page */
        constexpr u32 kPageNone = 0x3FFFFFFFu; /* answer's page when there is no run */
        constexpr u32 kPageSearch = 0x7FFFFFFFu; /* "use the lock-free search", not in the ring */
        constexpr u32 kServiceMaxPages = 1024u; /* 32 claims per lane, remembered in one word */
        constexpr u32 kServiceRetries = 4u; /* runs lost to chunk pages before the lock-free search is used */

        __host__ __device__ __forceinline__ mmc_page_service* page_service(mmc_heap_state* state)
        {
            return reinterpret_cast<mmc_page_service*>(state + 1);
        }

        /* longest run of set bits in x (31 for a full word; its callers treat full words apart) */
        __device__ __forceinline__ u32 longest_run(u32 x)
        {
            const u32 p1 = x & (x >> 1), p2 = p1 & (p1 >> 2), p3 = p2 & (p2 >> 4), p4 = p3 & (p3 >> 8);
            u32 cur = ~0u, len = 0u;
            if(p4 != 0u)
            {
                cur = p4;
                len = 16u;
            }
            u32 c = cur & (p3 >> len);
            if(c != 0u)
            {
                cur = c;
                len += 8u;
            }
            c = cur & (p2 >> len);
            if(c != 0u)
            {
                cur = c;
                len += 4u;
            }
            c = cur & (p1 >> len);
            if(c != 0u)
            {
                cur = c;
                len += 2u;
            }
            c = cur & (x >> len);
            return c != 0u ? len + 1u : len;
        }

        /* bits of word w that lie in pages [first, end) */
        __device__ __forceinline__ u32 word_span(u32 w, u32 first, u32 end)
        {
            const u32 lo = umax(first, 32u * w), hi = umin(end, 32u * w + 32u);
            if(lo >= hi)
                return 0u;
            const u32 n = hi - lo;
            return n == 32u ? 0xFFFFFFFFu : ((1u << n) - 1u) << (lo & 31u);
        }

        /* A kernel that calls malloc has the registers of its deepest call path,
         * taken or not. In one function the service took 103 to 124: a user's
         * kernel had two blocks of 256 threads per SM for four, and blocks of
         * 1024 threads were refused. So its steps are functions of their own (17
         * to 38 registers), called one after another from create, and what
         * lasts longer than a step lies in the kernel's stack frame (volatile:
         * read where it is used). malloc and free in a user's loop take 56
         * registers so, as without the service; with the steps called from a
         * function between them, 64 to 70. In a batch, a lane's word k has the
         * pages of requests 64 k + lane and 64 k + 32 + lane in its halves, 0
         * for none or placed. */
        constexpr u32 kServiceWords = 4u;
        constexpr u32 kServiceSlots = 2u * kServiceWords;
        constexpr u32 kServiceBatch = 32u * kServiceSlots;
        struct PageCall
        {
            PageScan c;
            /* the asking lane's */
            u32 bytes;
            u32 stage;
            u32 ticket;
            u32 polls;
            u32 seen; /* the tickets served, as lane 0 last saw them, */
            u32 idle; /* and how many looks ago that changed */
            u32 run; /* first page of the run found, kPageNone: none */
            /* the batch it serves */
            u32 head;
            u32 taken;
            u32 asked; /* which of the lane's words get an answer */
            u32 left; /* how many of them have no run yet */
            u32 entry; /* the hint as the batch found it */
            u32 w[kServiceWords];
            u32 page[kServiceSlots]; /* first pages of those placed */
        };
        /* A request that finds no run, or is served, is over; one that is too
         * large, or lost its runs to others, takes the lock-free search. */
        enum PageStage : u32
        {
            kAsks,
            kTicket, /* has a ticket, its word is not written yet */
            kWaits,
            kAnswered,
            kSearches,
            kOver
        };

        /* this lane's largest request of at most `fit` pages, 0: none */
        __device__ __forceinline__ u32 largest_request(const volatile PageCall& r, u32 fit)
        {
            const u32 f = umin(fit, 0xFFFFu);
            u32 most = 0u;
#pragma unroll
            for(u32 k = 0; k < kServiceWords; ++k)
            {
                const u32 v = r.w[k], lo = v & 0xFFFFu, hi = v >> 16;
                most = umax(most, umax(lo <= f ? lo : 0u, hi <= f ? hi : 0u));
            }
            return most;
        }

        /* one of this lane's requests of n pages gets its first page */
        __device__ __forceinline__ void place_request(volatile PageCall& r, u32 n, u32 page)
        {
            bool placed = false;
#pragma unroll 1
            for(u32 s = 0; !placed; ++s)
            {
                const u32 v = r.w[s / 2u], shift = 16u * (s & 1u);
                placed = ((v >> shift) & 0xFFFFu) == n;
                if(placed)
                {
                    r.w[s / 2u] = v & ~(0xFFFFu << shift);
                    r.page[s] = page;
                }
            }
            r.left = r.left - 1u;
        }

        /* the topmost run of n set bits of x, as the position of its lowest bit (there is one) */
        __device__ __forceinline__ u32 topmost_run(u32 x, u32 n)
        {
            for(u32 got = 1u; got < n && x != 0u;)
            {
                const u32 d = umin(got, n - got);
                x &= x >> d;
                got += d;
            }
            return 31u - static_cast<u32>(__clz(static_cast<int>(x)));
        }

        /* One pass of a batch's requests over the windows from page `top` down
         * to page `low` (both included), by a whole warp holding the lock. Returns
         * the highest page from which a later search could still find a
         * multi-page run. */
        __device__ __noinline__ inline u32 page_service_pass(volatile PageCall* call, u32 top, u32 low)
        {
            volatile PageCall& req = *call;
            u32* const freemap = req.c.freemap;
            constexpr u32 kFull = 0xFFFFFFFFu;
            const u32 lane = GpuIds::laneid();
            u32 hint = top;
            u32 carry = 0u; /* free pages right above the window */
            bool open = true; /* no usable run was left above */
            bool at_zero = false; /* a run was placed at page 0 */
            u32 w = top >> 10;
            u32 ahead[4];
#pragma unroll
            for(u32 k = 0; k < 4u; ++k)
                ahead[k] = (w >= k && 32u * (w - k) + lane <= req.c.numpages / 32u) ? ld_rlx(&freemap[32u * (w - k) + lane]) : 0u;
            for(;; --w)
            {
                u32 x = ahead[0] & word_span(32u * w + lane, low, top + 1u);
                ahead[0] = ahead[1];
                ahead[1] = ahead[2];
                ahead[2] = ahead[3];
                ahead[3] = w >= 4u ? ld_rlx(&freemap[32u * (w - 4u) + lane]) : 0u;
                MMC_STAT_ADD(req.c, MMC_STAT_PAGE_SCAN, 32u);
                if(__ballot_sync(kFull, x != 0u) == 0u)
                    carry = 0u;
                else
                {
                    for(;;)
                    {
                        const u32 t = static_cast<u32>(__clz(static_cast<int>(~x)));
                        const u32 notfull = __ballot_sync(kFull, x != kFull);
                        /* free pages right above this lane's word */
                        u32 above;
                        {
                            const u32 b = x == kFull ? 32u : static_cast<u32>(__ffs(static_cast<int>(~x))) - 1u;
                            const u32 higher = lane == 31u ? 0u : notfull >> (lane + 1u);
                            const u32 j = lane + static_cast<u32>(__ffs(static_cast<int>(higher))); /* lowest of them */
                            const u32 bj = __shfl_sync(kFull, b, static_cast<int>(j & 31u));
                            above = higher == 0u ? 32u * (31u - lane) + carry : 32u * (j - lane - 1u) + bj;
                        }
                        const u32 len = longest_run(x);
                        const u32 fit = __reduce_max_sync(kFull, umax(x != 0u ? above + t : 0u, len));
                        /* the largest waiting request that fits */
                        const u32 mine = largest_request(req, fit);
                        const u32 n = __reduce_max_sync(kFull, mine);
                        if(n == 0u)
                        {
                            /* to the next window: its carry, and what this one leaves */
                            if(open && fit > 1u)
                            {
                                /* the highest free page, or the stretch that joins this window's from above */
                                open = false;
                                const u32 hl = 31u - static_cast<u32>(__clz(static_cast<int>(__ballot_sync(kFull, x != 0u))));
                                const u32 th = 31u - static_cast<u32>(__clz(static_cast<int>(__shfl_sync(kFull, x, static_cast<int>(hl)))));
                                hint = 1024u * w + 32u * hl + th + (32u * hl + th == 1023u ? carry : 0u);
                            }
                            const u32 b = x == kFull ? 32u : static_cast<u32>(__ffs(static_cast<int>(~x))) - 1u;
                            const u32 l = static_cast<u32>(__ffs(static_cast<int>(notfull))) - 1u;
                            const u32 bl = __shfl_sync(kFull, b, static_cast<int>(l & 31u));
                            carry = notfull == 0u ? 1024u + carry : 32u * l + bl;
                            break;
                        }
                        /* its run: the topmost one */
                        const bool crossing = x != 0u && above + t >= n;
                        const u32 can = __ballot_sync(kFull, crossing || len >= n);
                        u32 q = 1024u * w + 32u * lane;
                        if(crossing)
                            q += 32u + above - n;
                        else if(len >= n)
                            q += topmost_run(x, n);
                        q = __shfl_sync(kFull, q, 31 - __clz(static_cast<int>(can)));
                        at_zero = at_zero || q == 0u;
                        const u32 used = word_span(32u * w + lane, q, q + n);
                        if(used != 0u)
                        {
                            x &= ~used;
                            atomicAnd(&freemap[32u * w + lane], ~used);
                        }
                        if(q + n > 1024u * w + 1024u)
                        {
                            /* the part above the window */
                            for(u32 ww = umax(32u * w + 32u, q >> 5) + lane; ww <= (q + n - 1u) >> 5; ww += 32u)
                                atomicAnd(&freemap[ww], ~word_span(ww, q, q + n));
                        }
                        if(q + n >= 1024u * w + 1024u)
                            carry = 0u; /* the pages above, if free, no longer join this window's */
                        if(lane == static_cast<u32>(__ffs(static_cast<int>(__ballot_sync(kFull, mine == n)))) - 1u)
                            place_request(req, n, q);
                    }
                }
                if(open)
                    hint = w == 0u ? 0u : umin(1024u * w - 1u, top);
                if(w == low >> 10 || !__any_sync(kFull, req.left != 0u))
                    break;
            }
            /* the reference stores a run's first page - 1, which wraps for a
             * run at page 0 (Scatter.hpp:800-804); fixed mode stores 0 */
            return at_zero && hint == 0u && req.c.reference_quirks ? 0xFFFFFFFFu : hint;
        }

        /* Pages (start - sum, start] all free, sum those of the batch's requests:
         * it packs there. (A run at page 0 is left to the passes.) */
        __device__ __noinline__ inline bool page_service_stretch(volatile PageCall* call, u32 sum)
        {
            constexpr u32 kFull = 0xFFFFFFFFu;
            volatile PageCall& req = *call;
            u32* const freemap = req.c.freemap;
            const u32 lane = GpuIds::laneid();
            const u32 start = umin(req.entry, req.c.numpages);
            if(sum >= start || start >= req.c.numpages)
                return false;
            const u32 low = start + 1u - sum;
            for(u32 w0 = start >> 5;; w0 -= 128u)
            {
                bool ok = true;
#pragma unroll
                for(u32 k = 0; k < 4u; ++k)
                {
                    const u32 off = 32u * k + lane;
                    const u32 w = w0 - off;
                    const u32 need = off <= w0 ? word_span(w, low, start + 1u) : 0u;
                    if(need != 0u)
                        MMC_STAT_ADD(req.c, MMC_STAT_PAGE_SCAN, 32u);
                    if(need != 0u)
                        ok = ok && (ld_rlx(&freemap[w]) & need) == need;
                }
                if(!__all_sync(kFull, ok))
                    return false;
                if(w0 < 128u || 32u * (w0 - 127u) <= low)
                    break;
            }
            for(u32 w = (low >> 5) + lane; w <= (start >> 5); w += 32u)
                atomicAnd(&freemap[w], ~word_span(w, low, start + 1u));
            u32 mine = 0u;
#pragma unroll
            for(u32 k = 0; k < kServiceWords; ++k)
            {
                const u32 v = req.w[k];
                mine += (v & 0xFFFFu) + (v >> 16);
            }
            u32 incl = mine;
#pragma unroll
            for(u32 off = 1u; off < 32u; off <<= 1)
            {
                const u32 v = __shfl_up_sync(kFull, incl, off);
                if(lane >= off)
                    incl += v;
            }
            u32 next = start + 1u - (incl - mine);
#pragma unroll
            for(u32 k = 0; k < kServiceWords; ++k)
            {
                const u32 v = req.w[k];
                next -= v & 0xFFFFu;
                req.page[2u * k] = next;
                next -= v >> 16;
                req.page[2u * k + 1u] = next;
                req.w[k] = 0u;
            }
            if(lane == 0u)
                atomicCAS(&req.c.state->firstFreePageBased, +req.entry, low - 1u);
            return true;
        }

        /* The next batch of the ring into the call's frame: the pages its
         * requests ask for, all told; 0 for an empty batch. A ticket drawn but
         * not written yet (its lane is about to) ends it. */
        __device__ __noinline__ inline u32 page_service_take(volatile PageCall* call)
        {
            constexpr u32 kFull = 0xFFFFFFFFu;
            volatile PageCall& req = *call;
            mmc_page_service* sv = page_service(req.c.state);
            const u32 lane = GpuIds::laneid();
            const u32 head = req.head;
            /* the words, read together with the tail: one a ticket has by then
             * and that holds no request yet is read again */
            u32 v[kServiceSlots];
#pragma unroll
            for(u32 s = 0; s < kServiceSlots; ++s)
                v[s] = ld_rlx(&sv->ring[(head + 32u * s + lane) & (MMC_PAGE_RING - 1u)]);
            const u32 have = __shfl_sync(kFull, umin(ld_rlx(&sv->tail) - head, kServiceBatch), 0);
            u32 taken = have;
#pragma unroll
            for(u32 s = 0; s < kServiceSlots; ++s)
            {
                const u32 i = 32u * s + lane;
#pragma unroll 1
                for(u32 spin = 0; i < taken && (v[s] & kPageAsk) == 0u; ++spin)
                {
                    v[s] = ld_rlx(&sv->ring[(head + i) & (MMC_PAGE_RING - 1u)]);
                    if(spin == 64u)
                        taken = i;
                }
                /* given up: kept as 0xFFFF until it is known whether the batch has it */
                v[s] = v[s] >= kPageGone ? 0xFFFFu : v[s] & 0xFFFFu;
                if((s & 1u) != 0u)
                    req.w[s / 2u] = v[s - 1u] | v[s] << 16;
            }
            taken = __reduce_min_sync(kFull, taken);
            u32 asked = 0u, sum = 0u;
#pragma unroll 1
            for(u32 s = 0; s < kServiceSlots; ++s)
            {
                const u32 w = req.w[s / 2u], shift = 16u * (s & 1u);
                const u32 n = (w >> shift) & 0xFFFFu, i = 32u * s + lane;
                const bool in = i < taken && n != 0xFFFFu;
                if(i < taken && n == 0xFFFFu)
                    st_rlx(&sv->ring[(head + i) & (MMC_PAGE_RING - 1u)], 0u);
                if(!in)
                    req.w[s / 2u] = w & ~(0xFFFFu << shift);
                asked |= in && n != 0u ? 1u << s : 0u;
                sum += in ? n : 0u;
            }
            req.taken = taken;
            req.asked = asked;
            req.left = static_cast<u32>(__popc(asked));
            return __reduce_add_sync(kFull, sum);
        }

        /* Answer the batch's requests (those placed have no pages left) and pass it. */
        __device__ __noinline__ inline void page_service_answer(volatile PageCall* call)
        {
            volatile PageCall& req = *call;
            mmc_page_service* sv = page_service(req.c.state);
            const u32 lane = GpuIds::laneid();
            const u32 head = req.head;
            /* every lane's bit clears are performed before any answer is seen */
            __threadfence();
            __syncwarp();
            u32 was[kServiceSlots];
            const u32 asked = req.asked;
#pragma unroll
            for(u32 s = 0; s < kServiceSlots; ++s)
            {
                const bool none = ((req.w[s / 2u] >> (16u * (s & 1u))) & 0xFFFFu) != 0u;
                const u32 answer = kPageAnswer | (none ? +kPageNone : +req.page[s]);
                was[s] = ((asked >> s) & 1u) != 0u
                    ? atomicExch(&sv->ring[(head + 32u * s + lane) & (MMC_PAGE_RING - 1u)], answer)
                    : 0u;
            }
            u32 gone = 0u; /* those whose askers have left since the batch was taken */
#pragma unroll
            for(u32 s = 0; s < kServiceSlots; ++s)
                if(was[s] >= kPageGone)
                {
                    /* (its half now says what goes back: the pages of a run that was placed) */
                    const u32 v = req.w[s / 2u], shift = 16u * (s & 1u);
                    req.w[s / 2u] = (v >> shift & 0xFFFFu) != 0u ? v & ~(0xFFFFu << shift) : v | (was[s] & 0xFFFFu) << shift;
                    gone |= 1u << s;
                }
#pragma unroll 1
            for(; gone != 0u; gone &= gone - 1u)
            {
                const u32 s = static_cast<u32>(__ffs(static_cast<int>(gone))) - 1u;
                const u32 n = (req.w[s / 2u] >> (16u * (s & 1u))) & 0xFFFFu;
                if(n != 0u)
                {
                    freemap_range(req.c.freemap, req.page[s], n, true);
                    atomicMax(&req.c.state->firstFreePageBased, req.page[s] + n - 1u);
                }
                st_rlx(&sv->ring[(head + 32u * s + lane) & (MMC_PAGE_RING - 1u)], 0u); /* idle again */
            }
            __syncwarp();
            req.head = head + req.taken;
            if(lane == 0u)
                st_rlx(&sv->head, head + req.taken);
        }

        /* The requests of a whole warp enter the ring: a ticket for each lane that asks. */
        __device__ __noinline__ inline bool page_service_enter(volatile PageCall* call)
        {
            const u32 asking = __ballot_sync(0xFFFFFFFFu, call->stage == kAsks);
            if(asking == 0u)
                return false;
            mmc_page_service* sv = page_service(call->c.state);
            u32 ticket = 0u;
            const u32 closed = __shfl_sync(0xFFFFFFFFu, ld_rlx(&sv->closed), 0);
            if(closed != 0u)
                return false;
            if(GpuIds::laneid() == 0u)
                ticket = atomicAdd(&sv->tail, static_cast<u32>(__popc(asking)));
            ticket = __shfl_sync(0xFFFFFFFFu, ticket, 0) + static_cast<u32>(__popc(asking & lanemask_lt()));
            if(call->stage == kAsks)
                call->stage = kTicket; /* (its run is kPageNone; the others' may have runs already) */
            call->ticket = ticket;
            call->polls = call->idle = call->seen = 0u;
            return true;
        }

        /* One look at the ring by a waiting warp: 0 when it waits no more, 1 to
         * look again, 2 when it has taken the lock to serve.
         *
         * A wait ends when no ticket has been served for MMC_SERVICE_MAX_IDLE
         * looks. (Not after a time of its own: a full grid's requests on a heap
         * that runs out wait for a thousand batches.) The warp that sees it
         * closes the service until the heap is initialised again; it and all
         * that wait give their requests up and search lock-free, as every later
         * request does. A ticket given up unwritten stays a hole in the ring,
         * which no server passes: hence the closing. A written word is given up
         * by a CAS, which fails when its answer is there. */
        __device__ __noinline__ inline u32 page_service_poll(volatile PageCall* call)
        {
            constexpr u32 kFull = 0xFFFFFFFFu;
            mmc_page_service* sv = page_service(call->c.state);
            const u32 ticket = call->ticket;
            u32* word = &sv->ring[ticket & (MMC_PAGE_RING - 1u)];
            u32 stage = call->stage;
            if(stage == kTicket)
            {
                /* a ticket's word is its own once the ticket a whole ring before
                 * it has been served and its answer read */
                if(ticket - ld_rlx(&sv->head) < MMC_PAGE_RING && ld_rlx(word) == 0u)
                {
                    st_rlx(word, kPageAsk | divup(call->bytes, call->c.pagesize));
                    stage = kWaits;
                }
            }
            else if(stage == kWaits)
            {
                const u32 v = ld_rlx(word);
                if((v & kPageAsk) == 0u)
                {
                    call->run = v & kPageNone;
                    st_rlx(word, 0u);
                    stage = kAnswered;
                }
            }
            u32 look = 0u; /* 1: again, 2: the lock is this warp's, 3: the service is closed */
            if(__any_sync(kFull, stage == kTicket || stage == kWaits))
            {
                look = 1u;
                if(GpuIds::laneid() == 0u)
                {
                    const u32 lock = ld_rlx(&sv->lock), head = ld_rlx(&sv->head), closed = ld_rlx(&sv->closed);
                    const u32 idle = head == call->seen ? call->idle + 1u : 0u;
                    call->seen = head;
                    call->idle = idle;
                    if(closed != 0u || idle > MMC_SERVICE_MAX_IDLE)
                    {
                        look = 3u;
                        if(atomicExch(&sv->closed, 1u) == 0u)
                            atomicOr(&call->c.state->error_flags, MMC_DEVERR_TIMEOUT);
                    }
                    else if(lock == 0u)
                        look = atomicCAS(&sv->lock, 0u, 1u) == 0u ? 2u : 1u;
                }
                look = __shfl_sync(kFull, look, 0);
                if(look == 3u)
                {
                    if(stage == kWaits)
                    {
                        const u32 asked = kPageAsk | divup(call->bytes, call->c.pagesize);
                        const u32 v = atomicCAS(word, asked, asked | kPageGone);
                        if(v != asked)
                        {
                            call->run = v & kPageNone;
                            st_rlx(word, 0u);
                            stage = kAnswered;
                        }
                    }
                    if(stage == kTicket || stage == kWaits)
                        stage = kSearches;
                    look = 0u;
                }
            }
            call->stage = stage;
            if(look == 1u)
            {
                const u32 polls = call->polls;
                call->polls = polls + 1u;
                if(polls > 1u)
                    __nanosleep(umin(64u << umin(polls, 5u), 1024u));
            }
            else /* the lock is taken, or answers are read: what servers did is performed before what follows */
                __threadfence();
            if(look == 2u)
                call->head = __shfl_sync(kFull, ld_rlx(&sv->head), 0);
            return look;
        }

        /* Serve what waits, batch by batch; the warp (whole) holds the lock. */
        __device__ __forceinline__ void page_service_run(volatile PageCall* call)
        {
#pragma unroll 1
            for(volatile u32 batch = 0; batch < 64u; batch = batch + 1u)
            {
                const u32 sum = page_service_take(call);
                if(call->taken == 0u)
                    break;
                /* one lane's reading for all: frees raise the hint meanwhile, and lanes
                 * with hints of their own clear bits of pages that no run has */
                call->entry = __shfl_sync(0xFFFFFFFFu, ld_rlx(&call->c.state->firstFreePageBased), 0);
                /* (from the reference's wrapped hint searches visit no page) */
                if(sum != 0u && call->entry != 0xFFFFFFFFu && !page_service_stretch(call, sum))
                {
                    /* from the hint down, then what is left from the top down to it */
                    const u32 hint = page_service_pass(call, umin(call->entry, call->c.numpages), 0u);
                    if(GpuIds::laneid() == 0u && hint != call->entry)
                        atomicCAS(&call->c.state->firstFreePageBased, +call->entry, hint);
                    if(__any_sync(0xFFFFFFFFu, call->left != 0u))
                        page_service_pass(call, call->c.numpages, umin(call->entry, call->c.numpages));
                }
                page_service_answer(call);
            }
            __threadfence();
            __syncwarp();
            if(GpuIds::laneid() == 0u)
                st_rlx(&page_service(call->c.state)->lock, 0u);
        }

        /* Claim the run that lane j was answered, a whole warp: 32 pages per
         * instruction. A run that is lost is given back, to be asked for again. */
        __device__ __noinline__ inline void claim_run_warp(volatile PageCall* call, int j)
        {
            constexpr u32 kFull = 0xFFFFFFFFu;
            volatile PageCall& req = *call;
            u32* const chunksize = req.c.chunksize;
            const u32 lane = GpuIds::laneid();
            const u32 first = __shfl_sync(kFull, req.run, j);
            const u32 tag = __shfl_sync(kFull, req.bytes, j);
            const u32 pages = divup(tag, req.c.pagesize);
            u32 got = 0u, lost = 0u;
#pragma unroll 4
            for(u32 i = 0; i < divup(pages, 32u); ++i)
            {
                const u32 off = 32u * i + lane;
                const u32 old = off < pages ? atomicCAS(&chunksize[first + off], 0u, tag) : 0u;
                got |= (off < pages && old == 0u ? 1u : 0u) << i;
                lost |= old;
            }
            const bool mine = lane == static_cast<u32>(j);
            if(!__any_sync(kFull, lost != 0u))
            {
                u32* wm = walkmap(req.c.freemap, req.c.numpages);
                for(u32 w = (first >> 5) + lane; 32u * w < first + pages; w += 32u)
                    atomicAnd(&wm[w], ~word_span(w, first, first + pages));
                __threadfence();
                if(mine)
                    req.stage = kOver;
                return;
            }
            /* A page of the run went to a chunk format or a lock-free
             * search: put the others back, as markpages does (each
             * lost page's owner keeps its bit). */
            MMC_STAT(req.c, MMC_STAT_PAGE_LOST);
            if(mine)
            {
                req.run = kPageNone;
                req.stage = kAsks;
            }
            u32 top = 0u;
#pragma unroll 1
            for(u32 m = got; m != 0u; m &= m - 1u)
            {
                const u32 page = first + 32u * (static_cast<u32>(__ffs(static_cast<int>(m))) - 1u) + lane;
                if(atomicCAS(&chunksize[page], tag, 0u) == tag)
                {
                    freemap_set(req.c.freemap, page);
                    top = page + 1u;
                }
            }
            if(top != 0u)
                atomicMax(&req.c.state->firstFreePageBased, top - 1u);
        }

        /* Multi-page requests of a whole warp, the call's bytes per lane, 0 for
         * none: the first page of the lane's run, claimed, kPageNone, or
         * kPageSearch where the lock-free search is to be used. */
        __device__ __forceinline__ u32 alloc_page_based_warp(volatile PageCall* call)
        {
            {
                const u32 n = divup(call->bytes, call->c.pagesize);
                call->stage = n == 0u ? kOver : (n <= kServiceMaxPages ? kAsks : kSearches);
                call->run = kPageNone;
            }
#pragma unroll 1
            for(volatile u32 round = 0; round < kServiceRetries && page_service_enter(call); round = round + 1u)
            {
                for(u32 look = 1u; look != 0u;)
                {
                    look = page_service_poll(call);
                    if(look == 2u)
                        page_service_run(call);
                }
                if(call->stage == kAnswered && call->run == kPageNone)
                {
                    MMC_STAT(call->c, MMC_STAT_PAGE_BASED_FAIL);
                    call->stage = kOver;
                }
                /* mark the runs, the warp together */
#pragma unroll 1
                for(volatile u32 todo = __ballot_sync(0xFFFFFFFFu, call->stage == kAnswered); todo != 0u;
                    todo = todo & (todo - 1u))
                    claim_run_warp(call, __ffs(static_cast<int>(todo)) - 1);
                __syncwarp();
            }
            return call->stage == kOver ? +call->run : +kPageSearch;
        }

        /* deallocPageBased, Scatter.hpp:874-886 (out of line, as the search) */
        __device__ __noinline__ inline void dealloc_page_based(const mmc_device_handle h, u32 page, u32 bytes)
        {
            const u32 pages = divup(bytes, h.pagesize);
            const u32 end = umin(page + pages, h.numpages);
            for(u32 p = page; p < end; ++p)
                page_init(h, p);
            freemap_range(walkmap(h.freemap, h.numpages), page, end - page, true);
            __threadfence();
            for(u32 p = page; p < end; ++p)
                atomicCAS(&h.chunksize[p], bytes, 0u);
            freemap_range(h.freemap, page, end - page, true);
            atomicMax(&h.state->firstFreePageBased, page + pages - 1u);
        }

        /* deallocPageBased for the lanes `runs` of the lanes `am`, which share
         * the work: a run's page tails, chunk sizes and bitmap words spread
         * over them. One lane alone zeroed 32 words per page and issued a
         * CAS per page: half of a wave's 920 blocks freed on a 512 MiB heap
         * took 202 us. Every lane's CASes are performed before any lane sets a
         * bit, by the fence and the barrier that all lanes pass: a bit set ahead
         * of its CAS could be taken by the server, whose claim then fails and
         * leaves the page's bit clear for good. */
        __device__ __noinline__ inline void dealloc_page_based_warp(const volatile PageScan* context, u32 masks, u32 am,
                                                                    u32 runs, u32 page, u32 bytes)
        {
            const volatile PageScan& c = *context;
            const u32 g = static_cast<u32>(__popc(am));
            const u32 rank = static_cast<u32>(__popc(am & lanemask_lt()));
            for(u32 todo = runs; todo != 0u; todo &= todo - 1u)
            {
                const int j = __ffs(static_cast<int>(todo)) - 1;
                const u32 first = __shfl_sync(am, page, j);
                const u32 tag = __shfl_sync(am, bytes, j);
                const u32 end = umin(first + divup(tag, c.pagesize), c.numpages);
                {
                    const u32 P = c.pagesize;
                    char* tail = c.pages + static_cast<u64>(first + 1u) * P - 4u * masks;
                    for(u32 p = first; p < end; ++p, tail += P)
                        for(u32 w = rank; w < masks; w += g)
                            st_rlx(reinterpret_cast<u32*>(tail) + w, 0u);
                }
                for(u32 w = (first >> 5) + rank; 32u * w < end; w += g)
                    atomicOr(&walkmap(c.freemap, c.numpages)[w], word_span(w, first, end));
                __threadfence();
                __syncwarp(am);
                u32* const chunksize = c.chunksize;
#pragma unroll 1
                for(u32 p = first + rank; p < end; p += g)
                    atomicCAS(&chunksize[p], tag, 0u);
                __threadfence();
                __syncwarp(am);
                for(u32 w = (first >> 5) + rank; 32u * w < end; w += g)
                    atomicOr(&c.freemap[w], word_span(w, first, end));
                if(rank == 0u)
                    atomicMax(&c.state->firstFreePageBased, first + divup(tag, c.pagesize) - 1u);
            }
        }

        /* create, Scatter.hpp:895-912, called by the lanes `active` together */
        template<class Ids>
        __device__ __forceinline__ void* create(const mmc_device_handle& h, u32 active, u32 bytes)
        {
            void* res = nullptr;
            const bool large = bytes > h.pagesize;
            const bool chunk = bytes != 0u && !large;
            if constexpr(Ids::warpSize > 1u)
            {
                /* chunks first: a warp's chunk requests need not wait for its
                 * multi-page ones, and in a heap that runs out they find their
                 * last chunks before the multi-page requests take the pages (a
                 * chunk request that finds none looks at every page, a
                 * multi-page one at a bit per page) */
                const u32 chunks = __ballot_sync(active, chunk);
                if(chunk)
                    res = alloc_chunked<Ids>(h, chunks, bytes);
                if constexpr(Ids::pageBased)
                {
                    if(__any_sync(active, large))
                    {
                        if(large)
                            MMC_STAT(h, MMC_STAT_PAGE_BASED);
                        const PageScan c{h.chunksize, h.freemap, h.state, h.pages, h.numpages, h.pagesize,
                                         h.reference_quirks};
                        u32 run = large ? kPageSearch : kPageNone;
                        /* a whole warp's are served together */
                        if(active == 0xFFFFFFFFu)
                        {
                            PageCall call;
                            call.c = c;
                            call.bytes = large ? bytes : 0u;
                            run = alloc_page_based_warp(&call);
                        }
                        if(run == kPageSearch)
                            res = alloc_page_based_concurrent(c, bytes);
                        else if(run != kPageNone)
                            res = page_data(h, run);
                    }
                }
                else if(large)
                    set_error(h, MMC_DEVERR_PAGEBASED);
            }
            else
            {
                if(chunk)
                    res = alloc_chunked<Ids>(h, active, bytes);
                else if(large)
                    res = alloc_page_based_single(h, bytes);
            }
            return res;
        }

        /* 64-bit division for page sizes that are not powers of two, kept out of line */
        __device__ __noinline__ inline u32 page_of_offset_slow(u64 offset, u32 pagesize)
        {
            return static_cast<u32>(offset / pagesize);
        }

        /* destroy, Scatter.hpp:918-946. A pointer outside the pool or on a page
         * without a chunk size (where the reference would divide by zero) is
         * recorded as MMC_DEVERR_BADFREE and ignored.
         *
         * Release: every access this thread made to the block is performed
         * before the atomics that hand the block to a next owner, by a release
         * fence ahead of them; the fence is cumulative, so it also covers what
         * other lanes of the warp did to the block before a __syncwarp this
         * thread passed (a warp-cooperative pattern's writes and reads). Every
         * lane fences before the lanes that free parts of one chunk meet at a
         * __syncwarp, so each lane's accesses to its part are performed before
         * the one grouped decrement. The reference's free has no such fence;
         * without it a thread's last reads of the block can be served after a
         * next owner's writes (a per-thread write/verify/free stress on GB300
         * read foreign data in 1 to 6 of 25 runs, none with the fence). */
        template<class Ids>
        __device__ void destroy(const mmc_device_handle& h, void* mem)
        {
            u32 active = 1u;
            if constexpr(Ids::warpSize > 1u)
                active = calling_lanes();
            const u32 P = h.pagesize;
            const u64 offset = static_cast<u64>(static_cast<char*>(mem) - h.pages);
            bool owned = mem != nullptr && offset < static_cast<u64>(h.numpages) * P;
            u32 page = 0u, chunksize = 0u;
            if(owned)
            {
                page = (P & (P - 1u)) == 0u ? static_cast<u32>(offset >> (__ffs(static_cast<int>(P)) - 1))
                                            : page_of_offset_slow(offset, P);
                /* The page's chunk size cannot change while this thread holds a
                 * block on it: it is loaded first, and its round trip overlaps the
                 * release fence's wait below instead of following it. */
                chunksize = ld_rlx(&h.chunksize[page]);
                release_fence();
            }
            if(mem != nullptr && chunksize == 0u)
                set_error(h, MMC_DEVERR_BADFREE);
            owned = chunksize != 0u;
            const u32 inpage_offset = static_cast<u32>(offset - static_cast<u64>(page) * P);
            const u32 block = owned ? inpage_offset / chunksize : 0u;
            const bool part = owned && inpage_offset != block * chunksize;
            const bool chunk = chunksize < P || (!h.reference_quirks && chunksize == P);
            u32 parts = 0u;
            bool runs = false; /* does any of the lanes free pages? (asked ahead of the count's round trip) */
            if constexpr(Ids::warpSize > 1u)
            {
                parts = __ballot_sync(active, part);
                runs = __any_sync(active, owned && !chunk);
            }
            if(part)
            {
                /* XMallocSIMD sub-allocation: the lane count lives at the chunk head.
                 * Lanes freeing parts of the same chunk together subtract as one
                 * (the lowest of them, after a __syncwarp that every lane
                 * reaches after its own release fence); whoever takes the count
                 * to zero frees the chunk, as each lane's own decrement would. */
                u32* counter = reinterpret_cast<u32*>(page_data(h, page) + block * chunksize);
                u32 sub = 1u;
                if constexpr(Ids::warpSize > 1u)
                {
                    const u32 peers = __match_any_sync(parts, reinterpret_cast<unsigned long long>(counter));
                    __syncwarp(peers);
                    sub = Ids::laneid() == static_cast<u32>(__ffs(static_cast<int>(peers))) - 1u
                        ? static_cast<u32>(__popc(peers))
                        : 0u;
                }
                owned = sub != 0u && atomicSub(counter, sub) == sub;
                mem = counter;
            }
            if constexpr(Ids::warpSize > 1u)
            {
                if(runs)
                {
                    const u32 which = __ballot_sync(active, owned && !chunk);
                    const PageScan c{h.chunksize, h.freemap, h.state, h.pages, h.numpages, h.pagesize, h.reference_quirks};
                    dealloc_page_based_warp(&c, h.maxOnPageMasks, active, which, page, chunksize);
                }
            }
            else if(owned && !chunk)
                dealloc_page_based(h, page, chunksize);
            if(owned && chunk)
                dealloc_chunked<Ids>(h, mem, page, chunksize);
        }

        /* OOM policy: ReturnNull::handleOOM (ReturnNull.hpp:48-51); MMC_OOM_FLAG
         * records the failure instead of BadAllocException's device assert. */
        template<class Ids>
        __device__ __forceinline__ void* handle_oom(const mmc_device_handle& h, void* mem, u32 req)
        {
            if(req != 0u && mem == nullptr && Ids::oom(h) == MMC_OOM_FLAG)
                set_error(h, MMC_DEVERR_OOM);
            return (req != 0u && mem == nullptr) ? nullptr : mem;
        }

        /* DeviceAllocator::malloc (device_allocator.hpp:72-82) with XMallocSIMD's
         * collect/distribute (XMallocSIMD.hpp:118-176): every active lane whose
         * padded size is in (0, pagesize/32) joins one allocation of
         * 16 + sum(sizes); the lowest such lane requests it, writes the lane
         * count at its head (the refcount destroy() decrements, Scatter.hpp:931-940)
         * and each lane receives base + 16 + (sizes of lower lanes). */
        template<class Ids>
        __device__ void* malloc(const mmc_device_handle& h, size_t bytes_in)
        {
            const u32 bytes = apply_padding(Ids::alignment(h), static_cast<u32>(bytes_in));
            /* one call of create for every form, so its code is in the kernel once */
            u32 req = bytes;
            u32 active = 1u;
            u32 joined = 0u; /* the lanes whose requests are one, 0: none are */
            u32 before = 0u;
            if constexpr(Ids::warpSize > 1u)
                active = calling_lanes();
            const u32 lane = Ids::laneid();
            if(Ids::coalesce && Ids::distribution(h) == MMC_DIST_XMALLOCSIMD)
            {
                const bool coalescible = bytes > 0u && bytes < (h.pagesize / 32u);
                joined = __ballot_sync(active, coalescible);
                joined = (joined & (joined - 1u)) != 0u ? joined : 0u;
                if(joined != 0u)
                {
                    /* exclusive prefix of the coalescible lanes' sizes, in lane order */
                    const u32 mine = coalescible ? bytes : 0u;
                    if(active == 0xFFFFFFFFu)
                    {
                        u32 incl = mine;
#pragma unroll
                        for(u32 off = 1u; off < 32u; off <<= 1)
                        {
                            const u32 v = __shfl_up_sync(0xFFFFFFFFu, incl, off);
                            if(lane >= off)
                                incl += v;
                        }
                        before = incl - mine;
                    }
                    else
                    {
#pragma unroll 1
                        for(u32 m = joined; m != 0u; m &= m - 1u)
                        {
                            const u32 src = static_cast<u32>(__ffs(static_cast<int>(m))) - 1u;
                            const u32 v = __shfl_sync(active, mine, static_cast<int>(src));
                            if(src < lane)
                                before += v;
                        }
                    }
                    const u32 total = __reduce_add_sync(active, mine);
                    if(coalescible)
                        req = (joined & lanemask_lt()) == 0u ? 16u + total : 0u; /* the lowest asks for all */
                }
            }
            void* mem = create<Ids>(h, active, req);
            mem = handle_oom<Ids>(h, mem, req);
            if constexpr(Ids::warpSize > 1u)
            {
                const bool part = ((joined >> lane) & 1u) != 0u;
                if(part && (joined & lanemask_lt()) == 0u && mem != nullptr)
                {
                    st_rlx(static_cast<u32*>(mem), static_cast<u32>(__popc(joined)));
                    /* The count's sector is usually cold, and the store leaves it
                     * partly valid in L2: the frees' atomics on it would wait for
                     * the DRAM fill. Fetch it now, while the lanes use their parts. */
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(mem));
                }
                /* The lane count must be seen by every later free of a sub-allocation
                 * (device-scope atomicSubs on this word). The warp barrier orders
                 * the leader's store before every lane's accesses after it, the
                 * frees included; a free by another thread is ordered through the
                 * synchronisation that handed it the pointer. (The reference stores
                 * the count with a block-scope fence, XMallocSIMD.hpp:160-166; a
                 * device-scope fence here measured 3-5 % slower on the batched
                 * workload.) It also brings the lanes together again after their
                 * searches. */
                __syncwarp(active);
                if(joined != 0u)
                {
                    const unsigned long long base = __shfl_sync(active, reinterpret_cast<unsigned long long>(mem),
                                                                __ffs(static_cast<int>(joined)) - 1);
                    if(part)
                        mem = base != 0ull ? reinterpret_cast<char*>(base) + 16u + before : nullptr;
                }
            }
            return mem;
        }

        template<class Ids>
        __device__ __forceinline__ void free(const mmc_device_handle& h, void* p)
        {
            destroy<Ids>(h, p);
        }

        /* For a caller about to free a block whose contents are dead: drop the
         * whole 128-byte lines inside [p, p + bytes) from L2 without writing
         * them back to DRAM (discard.global.L2; their bytes become
         * indeterminate), and return p, to be freed. Partial lines at the
         * ends are left alone (they may hold a neighbouring block). No
         * counterpart in the reference: a short-lived block's payload
         * otherwise costs a DRAM write-back after it is freed.
         *
         * Why no later owner's data can be discarded. In the PTX memory model
         * a discard is a weak write of indeterminate bytes to each line. The
         * free that follows issues a fence.release.gpu in every lane ahead of
         * the relaxed device-scope atomics that release the chunk, which
         * orders the discards (and every earlier access of the thread to the
         * block, including what other lanes of the warp wrote into it before a
         * __syncwarp this thread passed) before those atomics: a fence followed
         * by a strong write is a release pattern. A later owner can reach the block only
         * through an atomic that reads what those atomics wrote, and its
         * accesses to the block take their address from that atomic's result,
         * so they reach L2 after the discards. (A dependent read of each
         * discarded line, the other way to order them, misses L2 and measured
         * 17 % slower on the stress.) Call it right before the free. */
        __device__ __forceinline__ void* discard_dead_block(void* p, u32 bytes)
        {
            const u64 a = reinterpret_cast<u64>(p);
            const u64 lo = (a + 127ull) & ~127ull;
            const u64 end = a + bytes;
            for(u64 x = lo; x + 128ull <= end; x += 128ull)
                asm volatile("discard.global.L2 [%0], 128;" ::"l"(x) : "memory");
            return p;
        }

        /* ------------------------------------------------ free-slot counting */

        /* Run summary of a page range for the multi-page slot count: the
         * reference's serial scan (Scatter.hpp:1196-1217) counts
         * floor(L / pagestoalloc) per maximal run of L free pages; runs are
         * combined associatively so ranges can be scanned in parallel. */
        struct RunSum
        {
            u32 len; /* pages covered */
            u32 pre; /* free pages at the low end (== len if all free) */
            u32 suf; /* free pages at the high end */
            u32 cnt; /* slots in runs touching neither end */
        };

        __host__ __device__ __forceinline__ RunSum run_leaf(bool free_page)
        {
            return RunSum{1u, free_page ? 1u : 0u, free_page ? 1u : 0u, 0u};
        }
        __host__ __device__ __forceinline__ RunSum run_empty() { return RunSum{0u, 0u, 0u, 0u}; }

        /* a covers lower page indices than b */
        __host__ __device__ __forceinline__ RunSum run_combine(RunSum a, RunSum b, u32 n)
        {
            if(a.len == 0u)
                return b;
            if(b.len == 0u)
                return a;
            const bool af = a.pre == a.len;
            const bool bf = b.pre == b.len;
            RunSum r;
            r.len = a.len + b.len;
            if(af && bf)
            {
                r.pre = r.suf = r.len;
                r.cnt = 0u;
            }
            else if(af)
            {
                r.pre = a.len + b.pre;
                r.suf = b.suf;
                r.cnt = b.cnt;
            }
            else if(bf)
            {
                r.pre = a.pre;
                r.suf = a.suf + b.len;
                r.cnt = a.cnt;
            }
            else
            {
                r.pre = a.pre;
                r.suf = b.suf;
                r.cnt = a.cnt + b.cnt + (a.suf + b.pre) / n;
            }
            return r;
        }

        __host__ __device__ __forceinline__ u32 run_total(RunSum s, u32 n)
        {
            if(s.len != 0u && s.pre == s.len)
                return s.len / n;
            return s.cnt + s.pre / n + s.suf / n;
        }

        __device__ __forceinline__ RunSum shfl_runsum(u32 mask, RunSum s, int src)
        {
            RunSum r;
            r.len = __shfl_sync(mask, s.len, src);
            r.pre = __shfl_sync(mask, s.pre, src);
            r.suf = __shfl_sync(mask, s.suf, src);
            r.cnt = __shfl_sync(mask, s.cnt, src);
            return r;
        }

        /* Free slots of size slot on one page: getAvailaibleSlotsDeviceFunction's
         * single-page branch (Scatter.hpp:1164-1193) with countFreeChunksInPage
         * (:1112-1139). capZero = capacity at max(slot, paddedMinChunkSize). */
        __device__ __forceinline__ u32 page_free_slots(const mmc_device_handle& h, u32 chunksize, u32 count,
                                                       u32 slot, u32 maxchunksize, u32 slotChunk, u32 capSlotChunk)
        {
            if(chunksize >= slot && chunksize <= maxchunksize)
                return (chunksize == slotChunk ? capSlotChunk : page_capacity(h, chunksize)) - count;
            if(chunksize == 0u)
                return capSlotChunk - count;
            return 0u;
        }

        /* handle.getAvailableSlots (device_allocator.hpp:98-106 ->
         * getAvailableSlotsAccelerator, Scatter.hpp:1311-1352): the lanes active
         * at the call with one size share its scan and all of them receive the
         * count. Unlike the reference it needs no block-wide barrier, so any
         * subset of threads may call it; and lanes that come with different sizes
         * (also of one source line: the lanes of a loop meet in different rounds of
         * it) are parted first, where a scan over all of them would add up pages
         * counted for one size and the other. slotSize is padded first
         * (device_allocator.hpp:103). */
        template<class Ids>
        __device__ unsigned available_slots(const mmc_device_handle& h, size_t slotSize_in)
        {
            const u32 slot = apply_padding(Ids::alignment(h), static_cast<u32>(slotSize_in));
            if(slot == 0u)
                return 0u;
            u32 active = 1u, rank = 0u, nact = 1u;
            if(Ids::warpSize > 1u)
            {
                active = __match_any_sync(calling_lanes(), slot);
                nact = static_cast<u32>(__popc(active));
                rank = static_cast<u32>(__popc(active & lanemask_lt()));
            }
            const u32 P = h.pagesize;
            u32 partial = 0u;
            if(slot < P)
            {
                const u32 maxchunksize = umin(P, h.wastefactor * slot);
                const u32 slotChunk = umax(slot, h.paddedMinChunkSize);
                const u32 capSlotChunk = page_capacity(h, slotChunk);
                for(u32 pg = rank; pg < h.numpages; pg += nact)
                    partial += page_free_slots(h, ld_rlx(&h.chunksize[pg]), ld_rlx(&h.count[pg]), slot, maxchunksize,
                                               slotChunk, capSlotChunk);
                if(Ids::warpSize > 1u)
                    partial = __reduce_add_sync(active, partial);
                return partial;
            }
            /* multi-page slots: each active lane summarises a contiguous range,
             * the summaries are combined in lane order */
            const u32 n = divup(slot, P);
            const u32 per = divup(h.numpages, nact);
            const u32 b = umin(rank * per, h.numpages);
            const u32 e = umin(b + per, h.numpages);
            RunSum s = run_empty();
            for(u32 pg = b; pg < e; ++pg)
                s = run_combine(s, run_leaf(ld_rlx(&h.chunksize[pg]) == 0u), n);
            if(Ids::warpSize > 1u)
            {
                /* ordered fold over the active lanes, result broadcast */
                RunSum acc = run_empty();
                for(u32 m = active; m != 0u; m &= m - 1u)
                {
                    const int src = __ffs(static_cast<int>(m)) - 1;
                    acc = run_combine(acc, shfl_runsum(active, s, src), n);
                }
                s = acc;
            }
            return run_total(s, n);
        }
    } // namespace dev
} // namespace mmc
