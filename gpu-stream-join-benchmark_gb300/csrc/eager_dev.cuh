// eager_dev.cuh - device routines of the eager joins shared by the per-batch
// kernels (eager.cu) and the persistent eager kernel (eager_pk.cu): the
// side tables of the hash join and the searches of the sort-merge join.
#pragma once

#include "eager.cuh"

namespace sjbg {

constexpr uint32_t kNilIdx = 0xFFFFFFFFu;

struct ETab {
    uint32_t *keys, *cnt, *head, *next;
    unsigned long long *sum;
    uint32_t bits;
};

__device__ __forceinline__ int etab_lookup(const ETab &t, uint32_t key) {
    const uint32_t C = 1u << t.bits;
    if (key == kEmptyKey) return t.cnt[C] ? (int)C : -1;
    uint32_t s = slot_hash(key, t.bits);
    for (uint32_t p = 0; p < C; p++) {
        const uint32_t k = t.keys[s];
        if (k == key) return (int)s;
        if (k == kEmptyKey) return -1;
        s = (s + 1) & (C - 1);
    }
    return -1;
}

__device__ __forceinline__ unsigned long long own_hash(int side, uint32_t val) {
    return sjbg_fside(val, side == 0 ? 0u : 1u);
}

__device__ __forceinline__ void flush_batch(WinAcc *acc, unsigned long long *bcount, unsigned long long count,
                                            unsigned long long xr, unsigned long long prod) {
    flush_acc(acc, count, xr, prod);
    const unsigned long long c = warp_sum_u64(count);
    if (lane_id() == 0 && c) atomicAdd(bcount, c);
}

// A batch's matches on their way to the host.  Each CTA of the launch adds its
// count and one arrival to *sum in one atomic (the count in the low kCountBits,
// the arrivals above), so the last CTA to arrive holds the total without
// another trip to memory; it writes it to *host (mapped pinned memory) and
// leaves *sum zero for the next batch.  A count so costs no memset before the
// launch, no copy after it, and no fence.  wide: the batch may match 2^kCountBits
// pairs or has too many CTAs, so counts and arrivals go to words of their own.
constexpr uint32_t kCountBits = 48;
struct BatchCount {
    unsigned long long *sum;   // and sum[1]: the arrivals of a wide batch
    unsigned long long *host;
    bool wide;
};

// Adds the CTA's (count, xor, prod) to the window totals and publishes its
// count; called by every thread of a CTA of at most 256.
__device__ __forceinline__ void publish_batch(const BatchCount &bc, WinAcc *acc, unsigned long long count,
                                              unsigned long long xr, unsigned long long prod) {
    __shared__ unsigned long long part[3][8];
    count = warp_sum_u64(count);
    xr = warp_xor_u64(xr);
    prod = warp_sum_u64(prod);
    if (lane_id() == 0) {
        part[0][warp_id()] = count;
        part[1][warp_id()] = xr;
        part[2][warp_id()] = prod;
    }
    SJBG_BARRIER();
    if (threadIdx.x != 0) return;
    for (uint32_t w = 1; w < blockDim.x / 32; w++) {
        count += part[0][w];
        xr ^= part[1][w];
        prod += part[2][w];
    }
    if (!bc.wide) {
        const unsigned long long was = atomicAdd(bc.sum, count + (1ull << kCountBits));
        if ((was >> kCountBits) == gridDim.x - 1) {
            *bc.host = (was & ((1ull << kCountBits) - 1)) + count;
            *bc.sum = 0;
        }
    } else {
        atomicAdd(bc.sum, count);
        __threadfence();
        if (atomicAdd(bc.sum + 1, 1ull) == gridDim.x - 1) {
            __threadfence();
            *bc.host = atomicExch(bc.sum, 0ull);
            bc.sum[1] = 0;
        }
    }
    if (count) atomicAdd(&acc->count, count);
    if (xr) atomicXor(&acc->xr, xr);
    if (prod) atomicAdd(&acc->prod, prod);
}

// One incoming tuple of a hash-join batch (called by whole warps; `valid`
// false for the lanes past the batch): probe the other side's table (count
// and prod in O(1); the chain of the other side's tuple indices for the xor
// checksum and the pairs), then add the tuple, which sits at index `idx` of
// its side's tuple store, to its own side's table.  Adds the tuple's matches
// to count, xr and prod.  The two tables' first accesses go out together.
template <bool kEnum, bool kPairs>
__device__ __forceinline__ void eager_hj_step(bool valid, uint32_t key, uint32_t val, uint32_t idx, int side,
                                              const ETab &own, const ETab &oth, const sjbg_tuple *oth_tuples,
                                              uint32_t oth_n, WinAcc *acc, sjbg_pair *pairs, uint64_t pcap,
                                              unsigned long long &count, unsigned long long &xr,
                                              unsigned long long &prod) {
    const unsigned long long oh = own_hash(side, val);
    uint32_t head = kNilIdx, mine = 0;
    const uint32_t C = 1u << own.bits;
    uint32_t slot = C, held = key;   // the tuple's slot in its own table, and the key found there
    if (valid && key != kEmptyKey) {
        slot = slot_hash(key, own.bits);
        held = atomicCAS(&own.keys[slot], kEmptyKey, key);
    }
    if (valid) {
        const int s = etab_lookup(oth, key);
        if (s >= 0) {
            mine = oth.cnt[s];
            count += mine;
            prod += oh * oth.sum[s];
            if (kEnum || kPairs) head = oth.head[s];
        }
    }
    // chains hold indices of the other side's tuples; walks stop at its size
    if (kEnum) {
        uint32_t steps = 0;
        for (uint32_t j = head; j < oth_n && steps < oth_n; j = oth.next[j], steps++) {
            const uint32_t ov = oth_tuples[j].val;
            xr ^= side == 0 ? sjbg_pair_hash(val, ov) : sjbg_pair_hash(ov, val);
        }
    }
    if (kPairs) {
        uint32_t tot;
        const uint32_t ex = warp_excl_scan(mine, &tot);
        unsigned long long b = 0;
        if (lane_id() == 0 && tot) b = atomicAdd(&acc->npairs, (unsigned long long)tot);
        b = __shfl_sync(0xFFFFFFFFu, b, 0) + ex;
        uint32_t steps = 0;
        for (uint32_t j = head; j < oth_n && steps < oth_n; j = oth.next[j], b++, steps++) {
            const uint32_t ov = oth_tuples[j].val;
            if (b < pcap) pairs[b] = side == 0 ? sjbg_pair{val, ov} : sjbg_pair{ov, val};
        }
    }
    if (valid) {   // add the tuple to its own side's table
        for (uint32_t p = 1; held != kEmptyKey && held != key && p < C; p++) {   // (at most half full: a slot is found)
            slot = (slot + 1) & (C - 1);
            held = atomicCAS(&own.keys[slot], kEmptyKey, key);
        }
        atomicAdd(&own.cnt[slot], 1u);
        atomicAdd(&own.sum[slot], oh);
        // (only an enumerating handle walks the chains)
        if (kEnum || kPairs) own.next[idx] = atomicExch(&own.head[slot], idx);
    }
}

__device__ __forceinline__ uint32_t lower_bound_u32(const uint32_t *a, uint32_t n, uint32_t key) {
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (a[mid] < key) lo = mid + 1; else hi = mid;
    }
    return lo;
}
__device__ __forceinline__ uint32_t upper_bound_u32(const uint32_t *a, uint32_t n, uint32_t key) {
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (a[mid] <= key) lo = mid + 1; else hi = mid;
    }
    return lo;
}


}  // namespace sjbg
