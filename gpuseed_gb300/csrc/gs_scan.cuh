/*
 * gs_scan.cuh -- per-read counts into offsets, two counts at a time.
 *
 * A pass needs the offsets of its slots and work items before the search and
 * of its seeds and positions after it.  The kernel that makes the counts also
 * sums them by block, and the kernel that uses the offsets scans within its
 * block, so that the offsets take no launches of their own, which are most of
 * the time of a small pass: nine a pass in all, against 18 with device-wide
 * scans (one read 158 us instead of 228, 300 reads 300 instead of 354, 60,007
 * short reads 534 instead of 601; passes of milliseconds alike).  The totals
 * go to host memory as they are made.
 */
#ifndef GS_SCAN_CUH
#define GS_SCAN_CUH

#include "gs_internal.h"

#define GS_SCAN_THREADS 256u

/* reads [first, last) of block b of `blocks`: whole tiles of reads (at most
 * the block's threads), the same cut in both kernels */
__device__ __forceinline__ void gs_part_reads(uint32_t n, uint32_t tile, uint32_t b, uint32_t blocks,
                                              uint32_t &first, uint32_t &last)
{
    const uint32_t tiles = (n + tile - 1u) / tile;
    const uint32_t per = (tiles + blocks - 1u) / blocks;
    first = min(b * per * tile, n);
    last = min(first + per * tile, n);
}

/* exclusive sums of (a, b) over the block's threads; (ta, tb): the totals */
__device__ __forceinline__ GsPart gs_block_scan(unsigned long long a, unsigned long long b,
                                                GsPart &total)
{
    __shared__ GsPart s_warp[GS_SCAN_THREADS / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned long long ia = a, ib = b;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long x = __shfl_up_sync(0xffffffffu, ia, o);
        const unsigned long long y = __shfl_up_sync(0xffffffffu, ib, o);
        if (lane >= o) {
            ia += x;
            ib += y;
        }
    }
    __syncthreads();   /* the sums of the call before are read */
    if (lane == 31) {
        s_warp[w].a = ia;
        s_warp[w].b = ib;
    }
    __syncthreads();
    GsPart before = {0ull, 0ull};
    total.a = total.b = 0ull;
#pragma unroll
    for (int i = 0; i < (int)GS_SCAN_THREADS / 32; i++) {
        if (i == w) before = total;
        total.a += s_warp[i].a;
        total.b += s_warp[i].b;
    }
    before.a += ia - a;
    before.b += ib - b;
    return before;
}

/* Publishes the block's sums; the last block to do so turns all blocks' sums
 * into offsets and returns true with the totals. */
__device__ __forceinline__ bool gs_parts_publish(const GsParts &P, int which, GsPart sum, GsPart &total)
{
    __shared__ uint32_t s_last;
    if (threadIdx.x == 0) {
        P.part[blockIdx.x] = sum;
        __threadfence();
        s_last = atomicAdd(&P.tickets[which], 1u) == gridDim.x - 1u;
    }
    __syncthreads();
    if (!s_last) return false;
    __threadfence();
    /* a stretch of blocks a thread */
    const uint32_t per = (gridDim.x + GS_SCAN_THREADS - 1u) / GS_SCAN_THREADS;
    const uint32_t i0 = min(threadIdx.x * per, gridDim.x), i1 = min(i0 + per, gridDim.x);
    unsigned long long a = 0, b = 0;
#pragma unroll 8
    for (uint32_t i = i0; i < i1; i++) {
        a += __ldcg(&P.part[i].a);
        b += __ldcg(&P.part[i].b);
    }
    GsPart run = gs_block_scan(a, b, total);
#pragma unroll 8
    for (uint32_t i = i0; i < i1; i++) {
        GsPart v;
        v.a = __ldcg(&P.part[i].a);
        v.b = __ldcg(&P.part[i].b);
        P.part[i] = run;
        run.a += v.a;
        run.b += v.b;
    }
    if (threadIdx.x == 0) P.tickets[which] = 0u;
    return true;
}

#endif
