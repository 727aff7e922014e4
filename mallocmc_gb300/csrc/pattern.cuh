/* The workloads' payload: the u64 words m, m + 1, ... of a block, written and
 * read back 16 bytes at a time (chunks are 16-byte aligned under Shrink<16>). */
#pragma once

#include <cstdint>

/* Two u64 words at a (global, 16-byte aligned), where i < n; a load leaves
 * zeros elsewhere. Predicated by hand: as an if each became a branch with its
 * reconvergence. */
__device__ __forceinline__ void st_unit(uint64_t a, uint64_t x, uint64_t y, uint32_t i, uint32_t n)
{
    asm volatile("{.reg .pred p; setp.lt.u32 p, %3, %4; @p st.global.v2.u64 [%0], {%1, %2};}" ::"l"(a), "l"(x), "l"(y),
                 "r"(i), "r"(n)
                 : "memory");
}
__device__ __forceinline__ ulonglong2 ld_unit(uint64_t a, uint32_t i, uint32_t n)
{
    ulonglong2 v;
    asm volatile("{.reg .pred p; setp.lt.u32 p, %3, %4; mov.u64 %0, 0; mov.u64 %1, 0;"
                 " @p ld.global.v2.u64 {%0, %1}, [%2];}"
                 : "=&l"(v.x), "=&l"(v.y)
                 : "l"(a), "r"(i), "r"(n)
                 : "memory");
    return v;
}

/* The same for two units, four words from e, at a 32-byte aligned address. */
__device__ __forceinline__ void st_units2(uint64_t a, uint64_t e, uint32_t i, uint32_t n)
{
    asm volatile("{.reg .pred p; setp.lt.u32 p, %5, %6; @p st.global.v4.u64 [%0], {%1, %2, %3, %4};}" ::"l"(a), "l"(e),
                 "l"(e + 1u), "l"(e + 2u), "l"(e + 3u), "r"(i), "r"(n)
                 : "memory");
}
struct Units2
{
    uint64_t w[4];
};
__device__ __forceinline__ Units2 ld_units2(uint64_t a, uint32_t i, uint32_t n)
{
    Units2 v;
    asm volatile("{.reg .pred p; setp.lt.u32 p, %5, %6; mov.u64 %0, 0; mov.u64 %1, 0; mov.u64 %2, 0; mov.u64 %3, 0;"
                 " @p ld.global.v4.u64 {%0, %1, %2, %3}, [%4];}"
                 : "=&l"(v.w[0]), "=&l"(v.w[1]), "=&l"(v.w[2]), "=&l"(v.w[3])
                 : "l"(a), "r"(i), "r"(n)
                 : "memory");
    return v;
}

/* Write then verify the pattern of one thread's own block. Its lanes touch as
 * many cache lines per instruction as there are lanes, and one such sector
 * leaves the SM per cycle at most: 32 bytes a lane and instruction, a whole
 * sector, halve the requests of 16 (the first and the last unit go alone where
 * the block does not begin or end on a sector). A stress of blocks up to 2000
 * bytes took 3.05 ms with 16 bytes, 2.28 ms with 32. DEPTH pairs of units are
 * in flight in the read-back: two time as four, which spill. */
template<uint32_t DEPTH>
__device__ __forceinline__ void thread_pattern(char* ptr, uint32_t bytes, uint64_t m, uint32_t& bad,
                                               unsigned long long& csum)
{
    const uint32_t n16 = bytes / 16u;
    const uint64_t a = __cvta_generic_to_global(ptr);
    const uint32_t head = (static_cast<uint32_t>(a) >> 4) & (n16 != 0u ? 1u : 0u); /* units before the first pair */
    const uint32_t pairs = (n16 - head) / 2u;
    const uint32_t last = head + 2u * pairs; /* the unit after the pairs, if there is one */
    const uint64_t ap = a + 16u * head, mp = m + 2u * head;
    st_unit(a, m, m + 1u, 0u, head);
    st_unit(a + 16u * last, m + 2u * last, m + 2u * last + 1u, last, n16);
#pragma unroll 2
    for(uint32_t i = 0; i < pairs; ++i)
        st_units2(ap + 32u * i, mp + 4u * i, i, pairs);
    {
        const ulonglong2 f = ld_unit(a, 0u, head), l = ld_unit(a + 16u * last, last, n16);
        const uint64_t e = m + 2u * last;
        csum += (f.x ^ f.y) + (l.x ^ l.y);
        if(head != 0u)
            bad += (f.x != m) + (f.y != m + 1u);
        if(last < n16)
            bad += (l.x != e) + (l.y != e + 1u);
    }
#pragma unroll 1
    for(uint32_t i = 0; i < pairs; i += DEPTH)
    {
        Units2 v[DEPTH];
#pragma unroll
        for(uint32_t j = 0; j < DEPTH; ++j)
            v[j] = ld_units2(ap + 32u * (i + j), i + j, pairs);
        uint64_t diff = 0ull;
#pragma unroll
        for(uint32_t j = 0; j < DEPTH; ++j)
        {
            const uint64_t e = mp + 4u * (i + j);
            const uint64_t d = (v[j].w[0] ^ e) | (v[j].w[1] ^ (e + 1u)) | (v[j].w[2] ^ (e + 2u)) | (v[j].w[3] ^ (e + 3u));
            diff |= i + j < pairs ? d : 0ull;
            csum += (v[j].w[0] ^ v[j].w[1]) + (v[j].w[2] ^ v[j].w[3]);
        }
        if(diff != 0ull)
        {
#pragma unroll
            for(uint32_t j = 0; j < DEPTH; ++j)
            {
                const uint64_t e = mp + 4u * (i + j);
                if(i + j < pairs)
                    bad += (v[j].w[0] != e) + (v[j].w[1] != e + 1u) + (v[j].w[2] != e + 2u) + (v[j].w[3] != e + 3u);
            }
        }
    }
}

/* The verify workload's payload: n copies of the 32-bit word `value` from p
 * (4-byte aligned) on, written, or read back and the words that differ counted,
 * by one thread. Whole 32-byte sectors per access where the block has them: its
 * lanes' accesses fall in as many sectors as there are lanes, and word by word
 * each cost a request of its own (a million blocks of 8 to 600 bytes, one
 * kernel to allocate and one to verify and free: 968 -> 370 us). */
__device__ __forceinline__ void fill_words(uint32_t* p, uint32_t n, uint32_t value)
{
    const uint64_t a = __cvta_generic_to_global(p);
    const uint32_t head = min(static_cast<uint32_t>(0u - a) >> 2 & 7u, n); /* words before the first whole sector */
    const uint32_t sectors = (n - head) / 8u;
    const uint64_t two = static_cast<uint64_t>(value) << 32 | value;
    for(uint32_t i = 0; i < head; ++i)
        p[i] = value;
#pragma unroll 4
    for(uint32_t i = 0; i < sectors; ++i)
        asm volatile("st.global.v4.u64 [%0], {%1, %1, %1, %1};" ::"l"(a + 4u * head + 32u * i), "l"(two) : "memory");
    for(uint32_t i = head + 8u * sectors; i < n; ++i)
        p[i] = value;
}

__device__ __forceinline__ uint32_t wrong_words(const uint32_t* p, uint32_t n, uint32_t value)
{
    const uint64_t a = __cvta_generic_to_global(p);
    const uint32_t head = min(static_cast<uint32_t>(0u - a) >> 2 & 7u, n);
    const uint32_t sectors = (n - head) / 8u;
    const uint64_t two = static_cast<uint64_t>(value) << 32 | value;
    uint32_t bad = 0u;
    for(uint32_t i = 0; i < head; ++i)
        bad += p[i] != value;
#pragma unroll 1
    for(uint32_t i = 0; i < sectors; i += 4u)
    {
        Units2 v[4];
#pragma unroll
        for(uint32_t j = 0; j < 4u; ++j)
            v[j] = ld_units2(a + 4u * head + 32u * (i + j), i + j, sectors);
#pragma unroll
        for(uint32_t j = 0; j < 4u; ++j)
        {
            if(i + j >= sectors)
                continue;
            const uint64_t d[4] = {v[j].w[0] ^ two, v[j].w[1] ^ two, v[j].w[2] ^ two, v[j].w[3] ^ two};
            if((d[0] | d[1] | d[2] | d[3]) != 0ull)
#pragma unroll
                for(uint32_t k = 0; k < 4u; ++k)
                    bad += (static_cast<uint32_t>(d[k]) != 0u) + (static_cast<uint32_t>(d[k] >> 32) != 0u);
        }
    }
    for(uint32_t i = head + 8u * sectors; i < n; ++i)
        bad += p[i] != value;
    return bad;
}
