// range_join.cu - lazy counting joins by ranges, finished in shared memory (sm_103a).
//
// The counting form of the sort-merge join (smj.cu) when the windows' keys
// spread evenly enough: a most-significant-first sort that ends in shared
// memory.  The matching rule is the lazy CPU_SMJ's
// (src/sjb/windowing/lazy/executor/CPU/CPU_SMJ.cpp:23-139).
//   1. range_sample   per window: smallest and largest of a key sample -> a
//                     linear map of keys to P ranges (keys outside the
//                     sample's span fall into the end ranges: the map is
//                     monotone whatever the sample saw);
//   2. range_tiles    every tile of both sides sorted by range and written
//                     whole with its offsets (tiles.cuh);
//   3. range_join     persistent CTAs over the ranges: the left words of the
//                     range come into shared memory, distributed over its
//                     kRangeSubs equal subranges (a word or so each), and
//                     every right word meets the left words of its subrange.
//                     A range with a crowded subrange is sorted by the key
//                     bits in which its words differ, and its right words
//                     find their key groups by binary search: count += hi -
//                     lo, prod += gs * (F[hi] - F[lo]), F the prefix sums of fr.
// The tuples are read once, their words written and read once; the full radix
// sort reads and writes them three or four times, and the merge once more
// (128 windows of 2^10 to 2^20 tuples per side, keys in [0, 4 max(W)), 22.5 M
// tuples: 1.64 ms, and 0.55 by ranges).  A range that does not fit (hot or
// clustered keys) sets kErrRegroup, and the host makes the call again with the
// full sort.
//
// Hash joins of calls in the middle of the size range (hj.cu) take the same
// steps with ranges of a multiplicative hash of the key: no sample, two
// launches for the partitioning and the join, where counting, scanning and
// scattering first need five.  Counting, they add up the words of repeated keys
// in a table.
#include <algorithm>
#include <cstring>
#include <vector>

#include "sort.cuh"
#include "tiles.cuh"

namespace sjbg {

constexpr int kRangeThreads = 512;
constexpr int kRangeWarps = kRangeThreads / 32;
constexpr uint32_t kRangeCap = 4096;            // left words of a range (shared memory)
constexpr uint32_t kRangeWords = 8192;          // words of both sides
constexpr uint32_t kRangeTarget = 3328;         // left words per range, and half the words of both: uneven ranges still fit
// Fuller ranges, when they save a second wave of CTAs: up to here a range of
// keys with four tuples each has five standard deviations (sqrt(4 * 3,500) =
// 118) of room below kRangeCap, so some 304 ranges hardly ever miss.
constexpr uint32_t kRangeTargetMost = 3500;
constexpr uint32_t kRangesMax = 1024;           // more ranges: runs of under 4 words per tile
constexpr uint32_t kRangeTilesMax = 1536;       // tiles of both sides of a window
constexpr uint32_t kRangeDigit = 7;             // bits per shared-memory sorting pass
constexpr uint32_t kRangeDigits = 1u << kRangeDigit;
constexpr uint32_t kRangeSample = 8192;         // sampled keys per side
// The key map goes this many mean distances between sampled keys beyond the
// sample at each end.  Keys outside it fall into the end ranges, which have room
// for three such distances (of up to 256 left tuples each) above their share: one
// distance left out four in a hundred windows of 2^20 beside a small one, and 6
// in 60 draws of 128 windows of 2^10 to 2^20 took the sort, 1,640 us for 545.
// With eight none of 60 did; the other ranges get at most 1.6 % fuller.
constexpr uint32_t kRangeBeyond = 8;
constexpr uint32_t kRangeSubs = 2048;           // subranges of a range
// A range is crowded when one subrange holds more than kRangeCrowdMost left
// words or more than one thread in ten owns a subrange of more than
// kRangeCrowd: showing a few probes a few dozen words costs less than sorting
// the range (13 us; at a limit of 16 for every subrange, one range in 300 of
// keys with two duplicates each was sorted).
constexpr uint32_t kRangeCrowd = 16, kRangeCrowdMost = 128;
// By the hash, words of one subrange are mostly words of one key, so counting
// joins keep no list of a hot subrange, one with more than kRangeHot left words:
// they add up the words of each of its keys in a table behind the lists (with
// room for kRangeSubs words more than the lists need), and a probe looks there.
// When keys repeat throughout, every subrange is hot: with more than 3.5 left
// words that share a word's key on average, by the squares of the subranges'
// numbers (the rule of the bucket joins' places, hj.cu), and few enough keys for
// the table, by the subranges in use (kRangeUsed of 2,048: some 1,690 keys).
// 8 windows of 2^20, 1 / 2 / 4 / 8 / 16 / 64 tuples per key: lists, and a sort of
// crowded ranges, 238 / 253 / 281 / 335 / 449 / 627 us; hot subranges without the
// rule 246 / 261 / 293 / 348 / 370 / 222; with it 247 / 266 / 241 / 232 / 227 /
// 221.  Dense keys, z = 0.4 / 0.5: lists and sort 322 / 427, rule without hot
// subranges 322 / 430, both 277 / 297 (direct tables after radix partitioning 251
// / 252).  A kRangeHot of 4 / 8 / 12 / 20: distinct keys 392 / 287 / 250 / 246,
// z = 0.5 335 / 292 / 293 / 303.  A kRangeUsed of 1,350: one window of 1,000,003,
// z = 0.4 61 -> 82.  No room behind full lists, kRangeUsed 1,100: 500 windows of
// 20,000, z = 0.5 / 0.6 391 / 377 -> 456 / 543.  One window of 1,000,003 distinct
// keys pays 1 to 2 us of 57 for the rule and the table.
constexpr uint32_t kRangeHot = 16;
constexpr uint32_t kRangeRepeat2 = 7, kRangeUsed = 1150;
constexpr uint32_t kRangeHotBit = 1u << 31;   // of a subrange's first word: no list
constexpr uint32_t kRangeProbe = 64;   // slots of the table looked at for a key

struct RangeWin {
    uint64_t off[2], n[2];   // left, right
    uint32_t tile[2];        // first tile of the side
    uint32_t tiles[2];
    uint32_t bucket0, P;     // first range of the call, ranges
    uint64_t pairs_off, pairs_cap;
};

// The window's map of keys to ranges.
struct RangeMap {
    uint32_t lo, span, mult, P;   // span 0: every key in its own range, from lo
};

__device__ __forceinline__ uint32_t range_of(const RangeMap &m, uint32_t key) {
    const uint32_t d = key > m.lo ? key - m.lo : 0u, last = m.P - 1u;
    if (m.span == 0u) return min(d, last);
    return d >= m.span ? last : min(last, __umulhi(d, m.mult));
}

// Keys sampled from a side of n tuples: one in 256, at least 1,024, at most kRangeSample.
__device__ __forceinline__ uint64_t range_samples(uint64_t n) {
    return min(n, max((uint64_t)1024, min(n / 256, (uint64_t)kRangeSample)));
}

__global__ void __launch_bounds__(1024)
range_sample_kernel(const sjbg_tuple *__restrict__ L, const sjbg_tuple *__restrict__ R,
                    const RangeWin *__restrict__ wins, RangeMap *__restrict__ maps) {
    __shared__ uint32_t lo_s, hi_s;
    const RangeWin w = wins[blockIdx.x];
    if (threadIdx.x == 0) {
        lo_s = 0xFFFFFFFFu;
        hi_s = 0;
    }
    SJBG_BARRIER();
    uint32_t lo = 0xFFFFFFFFu, hi = 0;
#pragma unroll
    for (uint32_t side = 0; side < 2; side++) {
        const sjbg_tuple *src = (side ? R : L) + w.off[side];
        const uint64_t n = w.n[side], m = range_samples(n);
        uint32_t k[kRangeSample / 1024];
#pragma unroll
        for (uint32_t q = 0; q < kRangeSample / 1024; q++) {
            const uint64_t i = threadIdx.x + q * 1024;
            k[q] = i < m ? __ldg(&src[n == m ? i : i * n / m].key) : 0u;
        }
#pragma unroll
        for (uint32_t q = 0; q < kRangeSample / 1024; q++) {
            if (threadIdx.x + q * 1024 < m) {
                lo = min(lo, k[q]);
                hi = max(hi, k[q]);
            }
        }
    }
    lo = __reduce_min_sync(0xFFFFFFFFu, lo);
    hi = __reduce_max_sync(0xFFFFFFFFu, hi);
    if (lane_id() == 0) {
        atomicMin(&lo_s, lo);
        atomicMax(&hi_s, hi);
    }
    SJBG_BARRIER();
    if (threadIdx.x == 0) {
        RangeMap m;
        m.P = w.P;
        m.lo = 0;
        uint64_t span = 1;
        if (lo_s <= hi_s) {
            // the keys go a little beyond the sample's
            const uint64_t sampled = max(max(range_samples(w.n[0]), range_samples(w.n[1])), (uint64_t)64);
            const uint32_t more = (uint32_t)min(((uint64_t)hi_s - lo_s) * kRangeBeyond / sampled, (uint64_t)0xFFFFFFFFu);
            m.lo = lo_s > more ? lo_s - more : 0u;
            span = (uint64_t)(hi_s < 0xFFFFFFFFu - more ? hi_s + more : 0xFFFFFFFFu) - m.lo + 1;
        }
        if (span <= w.P) {
            m.span = m.mult = 0;
        } else {
            m.span = (uint32_t)(span > 0xFFFFFFFFull ? 0xFFFFFFFFull : span);
            m.mult = (uint32_t)(((uint64_t)w.P << 32) / span);   // P < span: below 2^32
        }
        maps[blockIdx.x] = m;
    }
}

// Range of a key: by the window's key map, or (hash) of the key's hash.
template <bool kHash>
struct RangeOf {
    RangeMap m;
    __device__ uint32_t operator()(uint32_t key) const {
        return kHash ? __umulhi(bucket_hash(key), m.P) : range_of(m, key);
    }
};

template <bool kHash>
__global__ void __launch_bounds__(kSortedThreads, 3)
range_tiles_kernel(const sjbg_tuple *__restrict__ L, const sjbg_tuple *__restrict__ R,
                   const RangeWin *__restrict__ wins, uint32_t nwin, uint32_t tiles, const RangeMap *__restrict__ maps,
                   uint32_t P, uint64_t *__restrict__ words, uint16_t *__restrict__ rows) {
    sort_tiles(tiles, [&](uint32_t tile, SortedTile &t) {
        uint32_t lo = 0, hi = nwin;   // largest w with tile[0] <= tile (a window's left tiles, then its right ones)
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (__ldg(&wins[mid].tile[0]) <= tile) lo = mid; else hi = mid;
        }
        const RangeWin &w = wins[lo];
        const uint32_t right = tile >= w.tile[1] ? 1u : 0u;
        const uint64_t start = (uint64_t)(tile - w.tile[right]) * kSortedTile, left = w.n[right] - start;
        RangeOf<kHash> f;
        if (kHash) f.m.P = w.P;
        else f.m = maps[lo];
        t.src = (right ? R : L) + w.off[right] + start;
        t.n = (uint32_t)(left < kSortedTile ? left : kSortedTile);
        t.P = f.m.P;
        t.words = words + (uint64_t)tile * kSortedTile;
        t.row = rows + (uint64_t)tile * sorted_row(P);   // (as long as the call's largest fan-out needs)
        return f;
    });
}

struct RangeTable {
    unsigned long long *sum;   // of fr
    uint32_t *key, *cnt;
    uint32_t slots;
};

struct RangeSmem {
    union {
        uint64_t word[kRangeCap + kRangeSubs];      // left words by subrange, and room for a table behind them
        uint32_t buf[2][2][kRangeCap];              // sorting: keys and vals, before and after a pass; then F in the free pair
    };
    union {
        uint32_t sub[kRangeSubs + 1];               // first left word of each subrange, and their number
        uint32_t wcnt[kRangeWarps][kRangeDigits + 1];   // sorting: per-warp digit counters (+ 1: no word)
    };
    uint32_t loc[kRangeDigits + 1];                 // first word of each digit of the last pass, and n
    uint16_t off[kRangeTilesMax], pre[kRangeTilesMax];   // per tile (left side's first): the run, the words before it
    uint16_t owner[kRangeWords];                    // tile of the range's i-th word
    uint32_t warp_tot[32], warp_used[32], warp_sq[32];
    unsigned long long wsum[32], base;
    uint32_t lo, hi, crowd, n_left, next, stop, refused;
};

// The slot of the table that holds the key or is the first free one from its
// home on; t.slots: neither among kRangeProbe slots.
__device__ __forceinline__ uint32_t range_slot(const RangeTable &t, uint32_t key) {
    uint32_t s = __umulhi(place_hash(key), t.slots);
    for (uint32_t p = 0; p < kRangeProbe; p++) {
        const uint32_t k = *(volatile const uint32_t *)&t.key[s];
        if (k == key || k == kEmptyKey) return s;
        s = s + 1 == t.slots ? 0u : s + 1;
    }
    return t.slots;
}

// Adds a left word to the table; false: no slot for its key (or the key is the
// mark of free slots).
__device__ __forceinline__ bool range_add(const RangeTable &t, uint64_t word) {
    const uint32_t key = (uint32_t)word;
    if (key == kEmptyKey) return false;
    for (;;) {   // (a slot lost to another key is taken for good: at most kRangeProbe times)
        const uint32_t s = range_slot(t, key);
        if (s == t.slots) return false;
        const uint32_t was = atomicCAS(&t.key[s], kEmptyKey, key);
        if (was != kEmptyKey && was != key) continue;
        atomicAdd(&t.cnt[s], 1u);
        ct_add_sum(&t.sum[s], sjbg_fr((uint32_t)(word >> 32)));
        return true;
    }
}

// One stable pass over the n left words in shared memory, on kRangeDigit bits
// of key - lo from `shift`.  Warp-private counters; a lane's digit peers come
// from one ballot per bit.
__device__ __forceinline__ void range_pass(RangeSmem &sm, uint32_t from, uint32_t n, uint32_t lo, uint32_t shift) {
    constexpr uint32_t kItems = kRangeCap / kRangeThreads;
    const uint32_t w = warp_id(), lane = lane_id();
    const uint32_t *keys = sm.buf[from][0], *vals = sm.buf[from][1];
    uint32_t *ko = sm.buf[from ^ 1][0], *vo = sm.buf[from ^ 1][1];
    for (uint32_t i = threadIdx.x; i < kRangeWarps * (kRangeDigits + 1); i += kRangeThreads) (&sm.wcnt[0][0])[i] = 0;
    SJBG_BARRIER();
    // warp w's positions [w * per, w * per + per), in order; per covers n evenly
    const uint32_t rounds = (n + kRangeThreads - 1) / kRangeThreads, first = w * rounds * 32;
    uint32_t rank[kItems], dig[kItems];
    const unsigned lt = (1u << lane) - 1u;
#pragma unroll
    for (uint32_t k = 0; k < kItems; k++) {
        if (k >= rounds) break;   // (the same for the whole CTA)
        const uint32_t pos = first + k * 32 + lane;
        const uint32_t d = pos < n ? ((keys[pos] - lo) >> shift) & (kRangeDigits - 1) : kRangeDigits;
        unsigned peers = 0xFFFFFFFFu;
#pragma unroll
        for (uint32_t b = 0; b <= kRangeDigit; b++) {
            const bool bit = (d >> b) & 1u;
            const unsigned m = __ballot_sync(0xFFFFFFFFu, bit);
            peers &= bit ? m : ~m;
        }
        const uint32_t cur = sm.wcnt[w][d];
        __syncwarp();
        rank[k] = cur + __popc(peers & lt);
        dig[k] = d;
        if (lane == (uint32_t)(__ffs(peers) - 1)) sm.wcnt[w][d] = cur + __popc(peers);
        __syncwarp();
    }
    SJBG_BARRIER();
    // per digit: exclusive over the warps, four threads per digit and four warps
    // per thread; then the digits' totals, by one warp
    {
        static_assert(kRangeThreads == 4 * kRangeDigits && kRangeWarps == 16, "four threads per digit");
        const uint32_t digit = threadIdx.x >> 2, q0 = (threadIdx.x & 3u) * 4;
        uint32_t c[4], sum = 0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            c[q] = sm.wcnt[q0 + q][digit];
            sum += c[q];
        }
        uint32_t run = sum;
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, run, o, 4);
            if ((threadIdx.x & 3u) >= (uint32_t)o) run += y;
        }
        if ((threadIdx.x & 3u) == 3u) sm.loc[digit] = run;
        run -= sum;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            sm.wcnt[q0 + q][digit] = run;
            run += c[q];
        }
    }
    SJBG_BARRIER();
    if (w == 0) {
        constexpr uint32_t kPer = kRangeDigits / 32;
        uint32_t a[kPer], sum = 0;
#pragma unroll
        for (uint32_t q = 0; q < kPer; q++) {
            a[q] = sm.loc[lane * kPer + q];
            sum += a[q];
        }
        uint32_t tot;
        uint32_t run = warp_excl_scan(sum, &tot);
#pragma unroll
        for (uint32_t q = 0; q < kPer; q++) {
            sm.loc[lane * kPer + q] = run;
            run += a[q];
        }
        if (lane == 31) sm.loc[kRangeDigits] = run;
    }
    SJBG_BARRIER();
#pragma unroll
    for (uint32_t k = 0; k < kItems; k++) {
        const uint32_t pos = first + k * 32 + lane;
        if (k < rounds && pos < n) {
            const uint32_t p = sm.loc[dig[k]] + sm.wcnt[w][dig[k]] + rank[k];
            ko[p] = keys[pos];
            vo[p] = vals[pos];
        }
    }
    SJBG_BARRIER();
}

// Exclusive prefix sums of fr over the range's n sorted words; returns their
// total to every thread; ends with a barrier.
__device__ __forceinline__ unsigned long long range_prefix(RangeSmem &sm, const uint32_t *vals, uint32_t n,
                                                           unsigned long long *F) {
    const uint32_t lane = lane_id(), wid = warp_id();
    const uint32_t rounds = (n + kRangeThreads - 1) / kRangeThreads, c0 = wid * rounds * 32;
    unsigned long long wtot = 0;
    for (uint32_t k = 0; k < rounds; k++) {
        const uint32_t i = c0 + k * 32 + lane;
        const unsigned long long f = i < n ? sjbg_fr(vals[i]) : 0ull;
        unsigned long long x = f;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= (uint32_t)o) x += y;
        }
        if (i < n) F[i] = wtot + x - f;   // within the warp's words
        wtot += __shfl_sync(0xFFFFFFFFu, x, 31);
    }
    if (lane == 0) sm.wsum[wid] = wtot;
    SJBG_BARRIER();
    const unsigned long long s = lane < kRangeWarps ? sm.wsum[lane] : 0ull;
    const unsigned long long base = warp_sum_u64(lane < wid ? s : 0ull), all = warp_sum_u64(s);
    for (uint32_t k = 0; k < rounds; k++) {   // each warp its own words
        const uint32_t i = c0 + k * 32 + lane;
        if (i < n) F[i] += base;
    }
    SJBG_BARRIER();
    return all;
}

// kEnum: every pair is visited for the xor checksum, kPairs: and written.
template <bool kHash, bool kEnum, bool kPairs>
__global__ void __launch_bounds__(kRangeThreads, 2)
range_join_kernel(const uint64_t *__restrict__ words, const uint16_t *__restrict__ rows,
                  const RangeWin *__restrict__ wins, uint32_t nwin, uint32_t nb, uint32_t P,
                  uint32_t *__restrict__ queue, WinAcc *__restrict__ acc, WinAcc *__restrict__ out,
                  sjbg_pair *__restrict__ pairs) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    RangeSmem &sm = *reinterpret_cast<RangeSmem *>(smem_raw);
    const uint32_t lane = lane_id(), wid = warp_id();
    uint32_t *status = reinterpret_cast<uint32_t *>(&acc[nwin].info);
    uint32_t g = blockIdx.x;   // the first range by position, the others from the queue
    while (g < nb) {
        uint32_t claim = 0;
        if (threadIdx.x == 0) {
            claim = gridDim.x + atomicAdd(queue, 1u);   // stored once this range is done
            sm.stop = *(volatile uint32_t *)status & kErrRegroup;
            sm.lo = 0xFFFFFFFFu;
            sm.hi = sm.crowd = sm.refused = 0;
        }
        uint32_t wlo = 0, whi = nwin;   // the range's window
        while (whi - wlo > 1) {
            const uint32_t mid = (wlo + whi) >> 1;
            if (__ldg(&wins[mid].bucket0) <= g) wlo = mid; else whi = mid;
        }
        const RangeWin &w = wins[wlo];
        const uint32_t TL = w.tiles[0], T = TL + w.tiles[1], tile0 = w.tile[0];   // (its right tiles follow its left ones)
        const uint16_t *rw = rows + (uint64_t)tile0 * sorted_row(P) + (g - w.bucket0);
        constexpr uint32_t kPerMax = kRangeTilesMax / kRangeThreads;
        const uint32_t per = (T + kRangeThreads - 1) / kRangeThreads, x0 = threadIdx.x * per;
        uint32_t len[kPerMax], sum = 0;
#pragma unroll
        for (uint32_t q = 0; q < kPerMax; q++) {
            const uint32_t x = x0 + q;
            len[q] = 0;
            if (q < per && x < T) {
                const uint16_t *r = rw + (uint64_t)x * sorted_row(P);
                const uint32_t o = __ldg(r);
                len[q] = __ldg(r + 1) - o;
                sm.off[x] = (uint16_t)o;
            }
            sum += len[q];
        }
        uint32_t tot;
        uint32_t run = warp_excl_scan(sum, &tot);
        if (lane == 31) sm.warp_tot[wid] = tot;
        SJBG_BARRIER();
        const uint32_t v = lane < kRangeWarps ? sm.warp_tot[lane] : 0u;
        const uint32_t n = __reduce_add_sync(0xFFFFFFFFu, v);
        run += __reduce_add_sync(0xFFFFFFFFu, lane < wid ? v : 0u);
        if (sm.stop || n > kRangeWords) {   // (the same for the whole CTA)
            if (threadIdx.x == 0) atomicOr(status, kErrRegroup);
            break;
        }
#pragma unroll
        for (uint32_t q = 0; q < kPerMax; q++) {
            const uint32_t x = x0 + q;
            if (q < per && x < T) {
                sm.pre[x] = (uint16_t)run;
                if (x == TL) sm.n_left = run;
                for (uint32_t m = 0; m < len[q]; m++) sm.owner[run + m] = (uint16_t)x;
            }
            run += len[q];
        }
        if (TL == T && threadIdx.x == 0) sm.n_left = n;
        SJBG_BARRIER();
        const uint32_t nl = sm.n_left;
        if (nl > kRangeCap) {   // (the same for the whole CTA)
            if (threadIdx.x == 0) atomicOr(status, kErrRegroup);
            break;
        }
        auto word = [&](uint32_t i) {
            const uint32_t x = sm.owner[i];
            return __ldg(words + (uint64_t)(tile0 + x) * kSortedTile + (sm.off[x] + (i - sm.pre[x])));
        };
        if (nl != 0 && nl != n) {
            // the left words, and the span of their keys
            constexpr uint32_t kItems = kRangeCap / kRangeThreads;
            uint64_t e[kItems];
            uint32_t klo = 0xFFFFFFFFu, khi = 0;
#pragma unroll
            for (uint32_t k = 0; k < kItems; k++) {
                const uint32_t i = threadIdx.x + k * kRangeThreads;
                e[k] = i < nl ? word(i) : 0ull;
            }
            for (uint32_t i = threadIdx.x; i <= kRangeSubs; i += kRangeThreads) sm.sub[i] = 0;
#pragma unroll
            for (uint32_t k = 0; k < kItems; k++) {
                if (threadIdx.x + k * kRangeThreads < nl) {
                    klo = min(klo, (uint32_t)e[k]);
                    khi = max(khi, (uint32_t)e[k]);
                }
            }
            klo = __reduce_min_sync(0xFFFFFFFFu, klo);
            khi = __reduce_max_sync(0xFFFFFFFFu, khi);
            if (lane == 0) {
                atomicMin(&sm.lo, klo);
                atomicMax(&sm.hi, khi);
            }
            SJBG_BARRIER();
            const uint32_t lo = sm.lo, hi = sm.hi;
            // the subrange of a key in [lo, hi] (the same rounding for every holder of the key)
            const float scale = (float)kRangeSubs / ((float)(hi - lo) + 1.0f);
            auto sub_of = [&](uint32_t key) {
                if (kHash) return place_hash(key) >> 21;
                return min(kRangeSubs - 1, (uint32_t)((float)(key - lo) * scale));
            };
            static_assert(kRangeSubs == 1u << 11, "sub_of takes 11 bits");
            uint32_t rank[kItems];
#pragma unroll
            for (uint32_t k = 0; k < kItems; k++)
                if (threadIdx.x + k * kRangeThreads < nl) rank[k] = atomicAdd(&sm.sub[sub_of((uint32_t)e[k])], 1u);
            SJBG_BARRIER();
            constexpr bool kTable = kHash && !kEnum;
            // by the hash a subrange's words are mostly one key's: the xor checksum visits all
            // of them either way (8 windows of 2^20, 16 tuples per key: 670 us, sorted 701;
            // written, the pairs of a sorted range take 1,013, else 1,069)
            constexpr bool kVisit = kHash && kEnum && !kPairs;
            bool crowded = false;
            [[maybe_unused]] RangeTable tab;
            {
                constexpr uint32_t kPer = kRangeSubs / kRangeThreads;
                uint32_t c[kPer], csum = 0, largest = 0, hot = 0;   // hot: bit q
                uint32_t used = 0, squares = 0;                     // (squares of at most kRangeCap words: 2^24)
#pragma unroll
                for (uint32_t q = 0; q < kPer; q++) {
                    c[q] = sm.sub[threadIdx.x * kPer + q];
                    largest = max(largest, c[q]);
                    if (kTable) {
                        used += c[q] != 0;
                        squares += c[q] * c[q];
                        if (c[q] > kRangeHot) {
                            hot |= 1u << q;
                            c[q] = 0;
                        }
                    }
                    csum += c[q];
                }
                uint32_t ctot;
                uint32_t crun = warp_excl_scan(csum, &ctot);
                if (kTable) {
                    used = __reduce_add_sync(0xFFFFFFFFu, used);
                    squares = __reduce_add_sync(0xFFFFFFFFu, squares);
                }
                if (lane == 31) {
                    sm.warp_tot[wid] = ctot;
                    if (kTable) {
                        sm.warp_used[wid] = used;
                        sm.warp_sq[wid] = squares;
                    }
                }
                if (kTable) {
                    SJBG_BARRIER();
                } else {
                    if (largest > kRangeCrowdMost) sm.crowd = 1;
                    crowded = __syncthreads_count(largest > (kVisit ? kRangeCrowdMost : kRangeCrowd)) > kRangeThreads / 10 || sm.crowd;
                }
                uint32_t v = lane < kRangeWarps ? sm.warp_tot[lane] : 0u;
                if (kTable) {
                    used = __reduce_add_sync(0xFFFFFFFFu, lane < kRangeWarps ? sm.warp_used[lane] : 0u);
                    squares = __reduce_add_sync(0xFFFFFFFFu, lane < kRangeWarps ? sm.warp_sq[lane] : 0u);
                    if (used <= kRangeUsed && 2 * (squares - nl * nl / kRangeSubs) > kRangeRepeat2 * nl) {   // no lists at all
                        hot = (1u << kPer) - 1;
                        v = crun = 0;
#pragma unroll
                        for (uint32_t q = 0; q < kPer; q++) c[q] = 0;
                    }
                }
                crun += __reduce_add_sync(0xFFFFFFFFu, lane < wid ? v : 0u);
#pragma unroll
                for (uint32_t q = 0; q < kPer; q++) {
                    sm.sub[threadIdx.x * kPer + q] = crun | (hot >> q & 1u ? kRangeHotBit : 0u);
                    crun += c[q];
                }
                if (threadIdx.x == kRangeThreads - 1) sm.sub[kRangeSubs] = crun;
                if constexpr (kTable) {
                    // the hot words' table: a slot for each of them, if there is room (half a slot there always is)
                    const uint32_t listed = __reduce_add_sync(0xFFFFFFFFu, v);
                    tab.slots = min((kRangeCap + kRangeSubs - listed) / 2, max(nl - listed, 64u));
                    tab.sum = reinterpret_cast<unsigned long long *>(sm.word + listed);
                    tab.key = reinterpret_cast<uint32_t *>(tab.sum + tab.slots);
                    tab.cnt = tab.key + tab.slots;
                    for (uint32_t i = threadIdx.x; listed < nl && i < tab.slots; i += kRangeThreads) {
                        tab.key[i] = kEmptyKey;
                        tab.cnt[i] = 0;
                        tab.sum[i] = 0;
                    }
                }
            }
            unsigned long long count = 0, prod = 0, xr = 0;
            // the right words one by one: first(x, j, end) gives the left words [j, end)
            // among which x's partners are, partner(x, j, lv) whether j is one and its val
            auto enumerate = [&](auto first, auto partner) {
                for (uint32_t i = nl + threadIdx.x; i < n; i += kRangeThreads) {
                    const uint64_t x = word(i);
                    const uint32_t rv = (uint32_t)(x >> 32);
                    uint32_t at, end, lv;
                    unsigned long long f = 0;
                    for (first(x, at, end); at < end; at++) {
                        if (!partner(x, at, lv)) continue;
                        count++;
                        f += sjbg_fr(lv);
                        xr ^= sjbg_pair_hash(lv, rv);
                    }
                    prod += f * sjbg_gs(rv);
                }
                if constexpr (kPairs) {
                    // one reservation for the range's pairs; each warp writes its own in turn, a
                    // pair of every lane that has one at a time, so that they lie side by side
                    // (8 windows of 2^20 with 1 / 4 / 16 tuples per key: 385 / 550 / 1,013 us, a
                    // lane's one after another 401 / 569 / 1,906)
                    uint32_t wt = (uint32_t)warp_sum_u64(count);
                    if (lane == 0) sm.warp_tot[wid] = wt;
                    SJBG_BARRIER();
                    const uint32_t c = lane < kRangeWarps ? sm.warp_tot[lane] : 0u;
                    const uint32_t total = __reduce_add_sync(0xFFFFFFFFu, c);
                    if (threadIdx.x == 0 && total)
                        sm.base = atomicAdd(&acc[wlo].npairs, (unsigned long long)total);
                    SJBG_BARRIER();
                    unsigned long long pos = sm.base + __reduce_add_sync(0xFFFFFFFFu, lane < wid ? c : 0u);
                    sjbg_pair *out_pairs = pairs + w.pairs_off;
                    for (uint32_t i0 = nl; total && i0 < n; i0 += kRangeThreads) {   // (whole warps step)
                        const uint32_t i = i0 + threadIdx.x;
                        const uint64_t x = i < n ? word(i) : 0ull;
                        uint32_t at = 0, end = 0, lv = 0;
                        if (i < n) first(x, at, end);
                        for (; __any_sync(0xFFFFFFFFu, at < end); at++) {
                            const bool has = at < end && partner(x, at, lv);
                            const unsigned m = __ballot_sync(0xFFFFFFFFu, has);
                            const unsigned long long mine = pos + __popc(m & ((1u << lane) - 1u));
                            if (has && mine < w.pairs_cap) out_pairs[mine] = sjbg_pair{lv, (uint32_t)(x >> 32)};
                            pos += __popc(m);
                        }
                    }
                }
            };
            if (!crowded) {
                SJBG_BARRIER();
#pragma unroll
                for (uint32_t k = 0; k < kItems; k++) {
                    if (threadIdx.x + k * kRangeThreads < nl) {
                        const uint32_t at = sm.sub[sub_of((uint32_t)e[k])];
                        if (kTable && (at & kRangeHotBit)) {
                            if (!range_add(tab, e[k])) sm.refused = 1;
                        } else {
                            sm.word[at + rank[k]] = e[k];
                        }
                    }
                    if (kTable) __syncwarp();
                }
                SJBG_BARRIER();
                if (kTable) crowded = sm.refused != 0;   // (sorted after all)
            }
            if (!crowded) {
                if constexpr (kEnum) {
                    enumerate(
                        [&](uint64_t x, uint32_t &j, uint32_t &end) {
                            const uint32_t key = (uint32_t)x;
                            j = end = 0;
                            if (key < lo || key > hi) return;
                            const uint32_t b = sub_of(key);
                            j = sm.sub[b];
                            end = sm.sub[b + 1];
                        },
                        [&](uint64_t x, uint32_t j, uint32_t &lv) {
                            const uint64_t y = sm.word[j];
                            lv = (uint32_t)(y >> 32);
                            return (uint32_t)y == (uint32_t)x;
                        });
                } else {
                    for (uint32_t i = nl + threadIdx.x; i < n; i += 4 * kRangeThreads) {
#pragma unroll
                        for (uint32_t q = 0; q < 4; q++)
                            e[q] = i + q * kRangeThreads < n ? word(i + q * kRangeThreads) : 0ull;
#pragma unroll
                        for (uint32_t q = 0; q < 4; q++) {
                            const uint32_t key = (uint32_t)e[q];
                            if (i + q * kRangeThreads >= n || key < lo || key > hi) continue;
                            const uint32_t b = sub_of(key), first = sm.sub[b], end = sm.sub[b + 1] & ~kRangeHotBit;
                            uint32_t c = 0;
                            unsigned long long f = 0;
                            if (kTable && (first & kRangeHotBit)) {
                                const uint32_t s = range_slot(tab, key);
                                if (s != tab.slots && tab.key[s] == key) {
                                    c = tab.cnt[s];
                                    f = tab.sum[s];
                                }
                            }
                            for (uint32_t j = first; j < end; j++) {   // (a hot subrange's first word is past any end)
                                const uint64_t x = sm.word[j];
                                if ((uint32_t)x == key) {
                                    c++;
                                    f += sjbg_fr((uint32_t)(x >> 32));
                                }
                            }
                            if (c) {
                                count += c;
                                prod += f * sjbg_gs((uint32_t)(e[q] >> 32));
                            }
                        }
                    }
                }
            } else {
#pragma unroll
                for (uint32_t k = 0; k < kItems; k++) {
                    const uint32_t i = threadIdx.x + k * kRangeThreads;
                    if (i < nl) {
                        sm.buf[0][0][i] = (uint32_t)e[k];
                        sm.buf[0][1][i] = (uint32_t)(e[k] >> 32);
                    }
                }
                SJBG_BARRIER();   // (sub is read by now: its space holds the sort's counters)
                const uint32_t bits = 32u - (uint32_t)__clz(hi - lo);   // (0: one key)
                uint32_t at = 0;   // the buffer pair that holds the words
                for (uint32_t shift = 0; shift < bits; shift += kRangeDigit, at ^= 1u) range_pass(sm, at, nl, lo, shift);
                const uint32_t *keys = sm.buf[at][0], *vals = sm.buf[at][1];
                // the key's group [l, h) among the words of its top digit
                const uint32_t shift = bits ? (bits - 1) / kRangeDigit * kRangeDigit : 0u;   // of the last pass
                auto group = [&](uint32_t key, uint32_t &l, uint32_t &h) {
                    l = h = 0;
                    if (key < lo || key > hi) return false;
                    uint32_t r = nl;
                    if (bits) {
                        const uint32_t digit = (key - lo) >> shift;
                        l = sm.loc[digit];
                        r = sm.loc[digit + 1];
                    }
                    const uint32_t end = r;
                    while (l < r) {
                        const uint32_t mid = (l + r) >> 1;
                        if (keys[mid] < key) l = mid + 1; else r = mid;
                    }
                    if (l >= end || keys[l] != key) return false;
                    h = l + 1;
                    r = end;
                    while (h < r) {
                        const uint32_t mid = (h + r) >> 1;
                        if (keys[mid] <= key) h = mid + 1; else r = mid;
                    }
                    return true;
                };
                if constexpr (kEnum) {
                    enumerate([&](uint64_t x, uint32_t &l, uint32_t &h) { if (!group((uint32_t)x, l, h)) l = h = 0; },
                              [&](uint64_t, uint32_t l, uint32_t &lv) {
                                  lv = vals[l];
                                  return true;
                              });
                } else {
                    unsigned long long *F = reinterpret_cast<unsigned long long *>(&sm.buf[at ^ 1][0][0]);
                    const unsigned long long all = range_prefix(sm, vals, nl, F);   // ends with a barrier
                    for (uint32_t i = nl + threadIdx.x; i < n; i += kRangeThreads) {
                        const uint64_t x = word(i);
                        uint32_t l, h;
                        if (!group((uint32_t)x, l, h)) continue;
                        count += h - l;
                        prod += ((h < nl ? F[h] : all) - F[l]) * sjbg_gs((uint32_t)(x >> 32));
                    }
                }
            }
            flush_acc(&acc[wlo], count, xr, prod);
        }
        if (threadIdx.x == 0) sm.next = claim;
        SJBG_BARRIER();
        g = sm.next;
        SJBG_BARRIER();   // read before the next claim is stored
    }
    // the last CTA to finish writes the results to pinned memory
    __threadfence();
    SJBG_BARRIER();
    if (threadIdx.x == 0) sm.stop = atomicAdd(queue + 1, 1u) == gridDim.x - 1 ? 1u : 0u;
    SJBG_BARRIER();
    if (!sm.stop) return;
    __threadfence();
    const unsigned long long *from = reinterpret_cast<const unsigned long long *>(acc);
    unsigned long long *to = reinterpret_cast<unsigned long long *>(out);
    for (uint32_t i = threadIdx.x; i < (nwin + 1) * (sizeof(WinAcc) / 8); i += kRangeThreads) to[i] = __ldcg(from + i);
}

static bool range_join_fits(const WinHost *wins, uint32_t n) {
    for (uint32_t w = 0; w < n; w++) {
        const uint64_t most = std::max(wins[w].n_left, wins[w].n_right);
        if (most > (uint64_t)kRangeTarget * kRangesMax) return false;
        if ((wins[w].n_left + kSortedTile - 1) / kSortedTile + (wins[w].n_right + kSortedTile - 1) / kSortedTile >
            kRangeTilesMax)
            return false;
    }
    return true;
}

int range_join_batch(sjbg_handle *h, const sjbg_tuple *dL, const sjbg_tuple *dR, const WinHost *wins, uint32_t n,
                     sjbg_pair *dPairs, WinAcc *hAcc, bool enumerate, bool hash) {
    std::vector<RangeWin> rw(n);
    const uint32_t slots = 2u * (uint32_t)std::max(h->num_sms, 1);   // resident CTAs of the join
    uint64_t tiles, nb;
    uint32_t pmax;
    auto plan = [&](uint32_t target) {
        tiles = nb = 0;
        pmax = 1;
        for (uint32_t w = 0; w < n; w++) {
            RangeWin &r = rw[w];
            std::memset(&r, 0, sizeof(r));
            r.off[0] = wins[w].left_off; r.n[0] = wins[w].n_left;
            r.off[1] = wins[w].right_off; r.n[1] = wins[w].n_right;
            r.pairs_off = wins[w].pairs_off;
            r.pairs_cap = dPairs ? wins[w].pairs_cap : 0;
            const bool empty = r.n[0] == 0 || r.n[1] == 0;   // (nothing of such a window is read)
            // by the left side, which a range holds whole, and by the words of both
            r.P = (uint32_t)std::max<uint64_t>({(r.n[0] + target - 1) / target,
                                                (r.n[0] + r.n[1] + 2 * target - 1) / (2 * target), 1});
            for (int s = 0; s < 2; s++) {
                r.tile[s] = (uint32_t)tiles;
                r.tiles[s] = empty ? 0u : (uint32_t)((r.n[s] + kSortedTile - 1) / kSortedTile);
                tiles += r.tiles[s];
            }
            r.bucket0 = (uint32_t)nb;
            nb += empty ? 0u : r.P;
            pmax = std::max(pmax, r.P);
        }
    };
    // ranges of a target (sides of at most kRangeTarget * kRangesMax tuples: 32 bits)
    auto ranges = [&](uint32_t target) {
        uint64_t sum = 0;
        for (uint32_t w = 0; w < n; w++) {
            const uint32_t l = (uint32_t)wins[w].n_left, r = (uint32_t)wins[w].n_right;
            if (l && r) sum += std::max({(l + target - 1) / target, (l + r + 2 * target - 1) / (2 * target), 1u});
        }
        return sum;
    };
    uint32_t target = kRangeTarget;
    if (hash && ranges(target) > slots && ranges(kRangeTargetMost) <= slots) {
        // about the least full ranges that make it one wave
        uint32_t no = target;
        for (target = kRangeTargetMost; target - no > 32;) {
            const uint32_t mid = (no + target) / 2;
            (ranges(mid) > slots ? no : target) = mid;
        }
    }
    plan(target);
    if (tiles > 0x7FFFFFFFull || nb > 0x7FFFFFFFull) return fail(h, SJBG_E_CAPACITY, "batch has too many tiles");
    if (nb == 0) {
        std::memset(hAcc, 0, sizeof(WinAcc) * (n + 1));
        return SJBG_OK;
    }
    // accumulators and status word, then the range queue and the count of finished CTAs
    const size_t upB = sizeof(RangeWin) * n, accB = (sizeof(WinAcc) * (n + 1) + 15) & ~(size_t)15;
    uint8_t *hst = static_cast<uint8_t *>(pinned_get(h, 0, upB));
    uint8_t *dev = static_cast<uint8_t *>(ws_get(h, WS_WIN_PLAN, upB));
    uint8_t *dAcc = static_cast<uint8_t *>(ws_get(h, WS_WIN_ACC, accB + 16));
    uint64_t *words = static_cast<uint64_t *>(ws_get(h, WS_SORT_K0, sizeof(uint64_t) * kSortedTile * tiles));
    uint16_t *rows = static_cast<uint16_t *>(ws_get(h, WS_SORT_HIST, sizeof(uint16_t) * sorted_row(pmax) * tiles));
    RangeMap *maps = static_cast<RangeMap *>(ws_get(h, WS_SORT_MAP, sizeof(RangeMap) * n));
    if (!hst || !dev || !dAcc || !words || !rows || !maps) return fail(h, SJBG_E_NOMEM, "range join buffers");
    WinAcc *acc = reinterpret_cast<WinAcc *>(dAcc);
    uint32_t *queue = reinterpret_cast<uint32_t *>(dAcc + accB);
    std::memcpy(hst, rw.data(), upB);
    if (int rc = stage_copy_zero(h, dev, hst, upB, dAcc, accB + 16)) return rc;
    const RangeWin *dW = reinterpret_cast<const RangeWin *>(dev);
    if (!hash)
        SJBG_CK(h, launch(h, "range_sample", range_sample_kernel, dim3(n), dim3(1024), 0, dL, dR, dW, maps));
    const size_t s1 = sorted_tile_bytes(pmax), s2 = sizeof(RangeSmem);
    auto tiles_kernel = hash ? range_tiles_kernel<true> : range_tiles_kernel<false>;
    allow_big_smem(tiles_kernel, s1);
    SJBG_CK(h, launch(h, "range_tiles", tiles_kernel,
                      dim3((uint32_t)std::min<uint64_t>(tiles, 3u * (uint64_t)std::max(h->num_sms, 1))),
                      dim3(kSortedThreads), s1, dL, dR, dW, n, (uint32_t)tiles, (const RangeMap *)maps, pmax, words,
                      rows));
    auto join_kernel = dPairs      ? (hash ? range_join_kernel<true, true, true> : range_join_kernel<false, true, true>)
                       : enumerate ? (hash ? range_join_kernel<true, true, false> : range_join_kernel<false, true, false>)
                                   : (hash ? range_join_kernel<true, false, false> : range_join_kernel<false, false, false>);
    allow_big_smem(join_kernel, s2);
    const uint32_t grid = (uint32_t)std::min<uint64_t>(nb, slots);
    SJBG_CK(h, launch(h, "range_join", join_kernel, dim3(grid), dim3(kRangeThreads), s2, (const uint64_t *)words,
                      (const uint16_t *)rows, dW, n, (uint32_t)nb, pmax, queue, acc, hAcc, dPairs));
    return SJBG_OK;
}

// Hash joins of the middle of the size range, when the choice is the library's.
// Below kHashLeast tuples one table per window has less to do (one window of
// 2^14 per side: 44.3 us against 45.9; of 2^16: 47.1 against 44.6).  Above
// kHashMost the bucket joins' time counts, not their launches (16 windows of
// 2^20: 433 us against 452; 64 of 2^18, keys in [0, W): 425 against 432, in
// [0, 4W): 493 against 396; 64 of 2^17: 256 against 235).
constexpr uint64_t kHashLeast = 1u << 17, kHashMost = 1u << 25;

// Many tiny windows whose other choice is an HBM table each: every window costs
// the ranges two tiles of the word array and a turn of a CTA (counting, W keys
// in [0, 4W): 16,000 windows of 16 tuples per side 1,200 us and 1 GB against
// 620 us and 21 MB; 512 of 1,000 92 against 80; 512 of 3,000 114 against 128,
// with keys in [0, W) 118 against 103).  Up to about a wave of CTAs the fixed
// costs decide, and the ranges' are lower (pairs, 128 of 1,000: 67 against 86).
constexpr uint64_t kHashMean = 6144;   // tuples of both sides per window

RouteTry &range_route(sjbg_handle *h, const WinHost *wins, uint32_t n) {
    uint64_t most = 0;
    for (uint32_t w = 0; w < n; w++) most = std::max({most, wins[w].n_left, wins[w].n_right});
    uint32_t bits = 0;
    for (; most; most >>= 1) bits++;
    return h->range_try[bits];
}

RangeScope::RangeScope(sjbg_handle *handle, const WinHost *wins, uint32_t n) : h(handle), t(range_route(handle, wins, n)) {
    h->use_ranges = t.open();
    h->by_ranges = h->held_back = false;
}

RangeScope::~RangeScope() {
    if (h->held_back && !once_missed) t.passed();
    h->use_ranges = h->by_ranges = h->held_back = false;
}

bool RangeScope::missed(unsigned long long status) {
    if (!h->by_ranges) return false;
    h->by_ranges = false;
    if (!(status & kErrRegroup)) {
        t.hit();
        return false;
    }
    t.miss();
    once_missed = true;
    h->use_ranges = false;
    return true;
}

bool range_join_pays(const sjbg_handle *h, const WinHost *wins, uint32_t n, bool enumerate) {
    if (n == 0 || h->cfg.algorithm == SJBG_ALG_NLJ) return false;
    if (h->cfg.algorithm == SJBG_ALG_HJ) {
        if (h->cfg.partitioner != SJBG_PART_AUTO || h->tune.partitioner) return false;
        uint64_t tuples = 0;
        for (uint32_t w = 0; w < n; w++) tuples += wins[w].n_left + wins[w].n_right;
        if (tuples < kHashLeast || tuples > kHashMost) return false;
        if (n > (enumerate ? 2u : 1u) * (uint32_t)std::max(h->num_sms, 1) && tuples < kHashMean * n &&
            choose_partitioner(h, wins, n) == SJBG_PART_NONE)
            return false;
    }
    return range_join_fits(wins, n);
}

}  // namespace sjbg
