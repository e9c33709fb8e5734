// tiles.cuh - tiles sorted by bucket: the partitioning step of the kernels that
// read a bucket's runs out of every tile (sm_103a).
//
// A tile of at most kSortedTile tuples is sorted by bucket in shared memory
// and written whole, as (val << 32 | key) words, to a region of its own, with
// a row of its buckets' offsets.  Nothing is counted beforehand and no global
// position is reserved: one read of the tuples, one coalesced write of half
// their bytes, no atomic outside shared memory.  A bucket is then the runs
// row[b] .. row[b + 1] of all tiles, in tile order; with P buckets a run has
// about kSortedTile / P words.
#pragma once

#include "runtime.h"

namespace sjbg {

constexpr uint32_t kSortedTile = 4096;
constexpr int kSortedThreads = 512;
constexpr int kSortedPer = kSortedTile / kSortedThreads;

// Row length in 16-bit words: offsets of P buckets and the end.
__host__ __device__ __forceinline__ uint32_t sorted_row(uint32_t P) { return (P + 8u) & ~7u; }

// Shared memory of sort_tile.
static inline size_t sorted_tile_bytes(uint32_t P) {
    return sizeof(uint64_t) * kSortedTile + sizeof(uint32_t) * (size_t)P;
}

// Multiplicative hash that picks a key's bucket (from its top bits), and the
// bits that spread a bucket's keys.  The second is not another multiple of the
// key: for dense keys the pairs of two multiples form a lattice, and one
// bucket's keys then crowd on a few places of the second.
__device__ __forceinline__ uint32_t bucket_hash(uint32_t key) { return key * 0x9E3779B1u; }
__device__ __forceinline__ uint32_t place_hash(uint32_t key) {
    const uint32_t h = bucket_hash(key);
    return (h ^ (h >> 13)) * 0x85EBCA6Bu;
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

// Where a tile's tuples lie and its sorted words and row go.
struct SortedTile {
    const sjbg_tuple *src;
    uint64_t *words;   // 16-byte aligned
    uint16_t *row;
    uint32_t n, P;     // n <= kSortedTile tuples, P buckets
};

// Sorts tiles blockIdx.x, blockIdx.x + gridDim.x, ... of `count`: tile_of(i, t)
// fills t and returns the tile's map of keys to buckets [0, P).  All
// kSortedThreads threads call it.  A tile's tuples are loaded while the one
// before it is written out (its registers are free by then), and are on their
// way into L2 before that.
template <typename TileOf>
__device__ __forceinline__ void sort_tiles(uint32_t count, TileOf tile_of) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ uint32_t warp_tot[32];
    uint64_t *stage = reinterpret_cast<uint64_t *>(smem_raw);
    uint32_t *cnt = reinterpret_cast<uint32_t *>(stage + kSortedTile);
    uint32_t it = blockIdx.x;
    if (it >= count) return;
    uint2 v[kSortedPer];
    auto load = [&](const SortedTile &t) {
#pragma unroll
        for (int k = 0; k < kSortedPer; k++) {
            const uint32_t i = threadIdx.x + k * kSortedThreads;
            v[k] = i < t.n ? __ldg(reinterpret_cast<const uint2 *>(t.src + i)) : make_uint2(0u, 0u);
        }
    };
    SortedTile t;
    auto bucket_of = tile_of(it, t);
    load(t);
    for (;;) {
        for (uint32_t i = threadIdx.x; i < t.P; i += kSortedThreads) cnt[i] = 0;
        SJBG_BARRIER();
        uint32_t br[kSortedPer];   // bucket << 16 | rank in the tile's bucket
#pragma unroll
        for (int k = 0; k < kSortedPer; k++)
            if (threadIdx.x + k * kSortedThreads < t.n) {
                const uint32_t b = bucket_of(v[k].x);
                br[k] = (b << 16) | atomicAdd(&cnt[b], 1u);
            }
        const uint32_t nit = it + gridDim.x;
        const bool more = nit < count;
        SortedTile nt = t;
        auto nbucket_of = bucket_of;
        if (more) {
            nbucket_of = tile_of(nit, nt);
            if (threadIdx.x == 0) l2_prefetch_bulk(nt.src, sizeof(sjbg_tuple) * nt.n);
        }
        SJBG_BARRIER();
        tile_scan(cnt, t.P, warp_tot);
#pragma unroll
        for (int k = 0; k < kSortedPer; k++)
            if (threadIdx.x + k * kSortedThreads < t.n)
                stage[cnt[br[k] >> 16] + (br[k] & 0xFFFFu)] = ((uint64_t)v[k].y << 32) | v[k].x;
        for (uint32_t i = threadIdx.x; i < t.P; i += kSortedThreads) t.row[i] = (uint16_t)cnt[i];
        if (threadIdx.x == 0) t.row[t.P] = (uint16_t)t.n;
        if (more) load(nt);
        SJBG_BARRIER();
        const uint4 *s4 = reinterpret_cast<const uint4 *>(stage);
        for (uint32_t i = threadIdx.x; i < t.n / 2; i += kSortedThreads) reinterpret_cast<uint4 *>(t.words)[i] = s4[i];
        if ((t.n & 1u) && threadIdx.x == 0) t.words[t.n - 1] = stage[t.n - 1];
        if (!more) return;
        it = nit;
        t = nt;
        bucket_of = nbucket_of;
    }
}

}  // namespace sjbg
