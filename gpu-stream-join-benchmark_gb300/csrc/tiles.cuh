// tiles.cuh - tiles sorted by bucket: the partitioning step of the kernels that
// read a bucket's runs out of every tile (sm_103a).
//
// A tile of at most kSortedTile tuples is sorted by bucket in shared memory
// and written whole, as (val << 32 | key) words, to a region of its own, with
// a row of its buckets' offsets.  Nothing is counted beforehand and no global
// position is reserved: one read of the tuples, one coalesced write of half
// their bytes, no atomic outside shared memory.  A bucket is then the runs
// row[b] .. row[b + 1] of all tiles, in tile order; with 2^lg buckets a run
// has about kSortedTile / 2^lg words.
#pragma once

#include "runtime.h"

namespace sjbg {

constexpr uint32_t kSortedTile = 4096;
constexpr int kSortedThreads = 512;
constexpr int kSortedPer = kSortedTile / kSortedThreads;

// Row length in 16-bit words: offsets of 2^lg buckets and the end, 16-byte rows.
__host__ __device__ __forceinline__ uint32_t sorted_row(uint32_t lg) { return (1u << lg) + 8u; }

// Shared memory of sort_tile.
static inline size_t sorted_tile_bytes(uint32_t lg) {
    return sizeof(uint64_t) * kSortedTile + sizeof(uint32_t) * (size_t)(1u << lg);
}

// Block-wide exclusive scan of P shared counters in place.
__device__ __forceinline__ void tile_scan(uint32_t *a, uint32_t P, uint32_t *warp_tot) {
    const uint32_t per = (P + blockDim.x - 1) / blockDim.x;
    const uint32_t b0 = min(P, threadIdx.x * per), b1 = min(P, b0 + per);
    uint32_t s = 0;
    for (uint32_t i = b0; i < b1; i++) s += a[i];
    uint32_t tot;
    const uint32_t ex = warp_excl_scan(s, &tot);
    if (lane_id() == 31) warp_tot[warp_id()] = ex + s;
    SJBG_BARRIER();
    if (warp_id() == 0) {
        const uint32_t x = lane_id() < (blockDim.x >> 5) ? warp_tot[lane_id()] : 0u;
        uint32_t tt;
        warp_tot[lane_id()] = warp_excl_scan(x, &tt);
    }
    SJBG_BARRIER();
    uint32_t run = warp_tot[warp_id()] + ex;
    for (uint32_t i = b0; i < b1; i++) {
        const uint32_t c = a[i];
        a[i] = run;
        run += c;
    }
    SJBG_BARRIER();
}

// Sorts the n <= kSortedTile tuples at src by bucket_of(key) in [0, 2^lg) into
// words[0 .. n) (16-byte aligned) and writes their row.  All kSortedThreads
// threads call it.
template <typename BucketOf>
__device__ __forceinline__ void sort_tile(const sjbg_tuple *__restrict__ src, uint32_t n, uint32_t lg,
                                          uint64_t *__restrict__ words, uint16_t *__restrict__ row,
                                          BucketOf bucket_of) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ uint32_t warp_tot[32];
    uint64_t *stage = reinterpret_cast<uint64_t *>(smem_raw);
    uint32_t *cnt = reinterpret_cast<uint32_t *>(stage + kSortedTile);
    const uint32_t P = 1u << lg;
    uint2 v[kSortedPer];
#pragma unroll
    for (int k = 0; k < kSortedPer; k++) {
        const uint32_t i = threadIdx.x + k * kSortedThreads;
        v[k] = i < n ? __ldg(reinterpret_cast<const uint2 *>(src + i)) : make_uint2(0u, 0u);
    }
    for (uint32_t i = threadIdx.x; i < P; i += kSortedThreads) cnt[i] = 0;
    SJBG_BARRIER();
    uint32_t rank[kSortedPer];
#pragma unroll
    for (int k = 0; k < kSortedPer; k++)
        if (threadIdx.x + k * kSortedThreads < n) rank[k] = atomicAdd(&cnt[bucket_of(v[k].x)], 1u);
    SJBG_BARRIER();
    tile_scan(cnt, P, warp_tot);
#pragma unroll
    for (int k = 0; k < kSortedPer; k++)
        if (threadIdx.x + k * kSortedThreads < n)
            stage[cnt[bucket_of(v[k].x)] + rank[k]] = ((uint64_t)v[k].y << 32) | v[k].x;
    for (uint32_t i = threadIdx.x; i < P; i += kSortedThreads) row[i] = (uint16_t)cnt[i];
    if (threadIdx.x == 0) row[P] = (uint16_t)n;
    SJBG_BARRIER();
    const uint4 *s4 = reinterpret_cast<const uint4 *>(stage);
    for (uint32_t i = threadIdx.x; i < n / 2; i += kSortedThreads) reinterpret_cast<uint4 *>(words)[i] = s4[i];
    if ((n & 1u) && threadIdx.x == 0) words[n - 1] = stage[n - 1];
}

}  // namespace sjbg
