// hj.cu - lazy hash join (sm_103a).
//
// Replaces the reference's lazy GPU hash-join family
// (src/sjb/windowing/lazy/executor/GPU/GPU_HJ.cu:9-309 and its NoOutput /
// CountKernel / EstimatedSelectivity / Atomic variants), whose matching rule
// is the lazy CPU_HJ's (src/sjb/windowing/lazy/executor/CPU/CPU_HJ.cpp:30-136):
// every left tuple joins every right tuple of the window with an equal key.
//
// Design (many windows per call, one launch per pass):
//   1. part_hist     per 4096-tuple tile: bucket of each tuple -> shared histogram
//                    -> one atomicAdd per non-empty bucket into the global counts.
//   2. part_scan     per window, exclusive scan of its counts on both sides ->
//                    bucket starts; buckets with tuples on both sides form the
//                    join list: the smaller run builds, a long probe run is cut
//                    in pieces, and both runs of a bucket far longer than its
//                    table are.  A window whose smaller side is one bucket is
//                    not partitioned: its pieces read the tuples themselves.
//   3. part_scatter  per tile: local counting sort by bucket in shared memory,
//                    one atomicAdd per bucket to reserve a range, then the tile
//                    is written as contiguous per-bucket runs of (key,val) words
//                    (windows of many buckets: a coarse pass inside part_hist,
//                    then part_fine).  A learned window's compacted light tuples
//                    are only sorted by bucket inside their tiles (part_light),
//                    and the join takes a bucket's runs out of all tiles.
//   4. bucket_join   per join item (persistent CTAs, one item ahead): a radix
//                    bucket through a direct table indexed by key >> radix bits
//                    when its indices allow it, else by places (short lists by
//                    a hash of the key), else through an open-addressing table,
//                    as learned buckets; built from the build run, probed with
//                    the other.
//        count mode: table slot = {key, count, hash sum}, updated with
//                    32-bit shared atomics (the sum as two words with carry);
//                    keys that do not fit go back into the build run (compacted
//                    in place) and are joined in a further pass, so any bucket,
//                    however skewed, finishes.
//        enum mode:  table slot = {key, chain head}, chains over a staged chunk
//                    of left vals; every pair is visited for the xor checksum
//                    and, when asked, written with one atomic per warp.
// The bucket of a key is its low radix bits (plain radix partitioning) or the
// learned partitioner's prediction (learned.cu).
// Counting calls of small windows only take one launch (hj_raw_batch), and
// those of the middle of the size range go by hash ranges (range_join.cu).
#include <algorithm>
#include <cstring>
#include <type_traits>
#include <vector>

#include "learned.cuh"
#include "runtime.h"
#include "tiles.cuh"

namespace sjbg {

constexpr int kTile = 4096;          // tuples per partitioning tile
constexpr uint32_t kHistTiles = 16;  // tiles per counting CTA at least with a model (amortises its set-up)
constexpr int kPartThreads = 512;
constexpr int kJoinThreads = 512;
constexpr uint32_t kMaxBucketsLog2 = 14;
// Two-level partitioning: a window of 2^lg buckets is split into 2^ceil(lg/2)
// coarse partitions of 2^floor(lg/2) fine buckets each (at most 128 of each).
constexpr uint32_t kCoarseMax = 128;
constexpr uint32_t kRow = kCoarseMax + 1;   // per tile: exclusive coarse offsets, then its total
constexpr uint32_t kGroupTiles = 64;        // tiles whose runs of one coarse partition a fine CTA gathers
// Tuples a fine CTA sorts at a time.  An item of a window that is half light
// has 2,048 tuples on average and an all-light one 4,096, so chunks hold a
// quarter more: at 2,048 every second item had a chunk of a few tuples.
constexpr uint32_t kFineChunk = 2560;
constexpr int kFineThreads = 256;

__host__ __device__ __forceinline__ uint32_t coarse_bits(uint32_t lg) { return (lg + 1) / 2; }
// Windows of at least this many buckets are partitioned in two passes: with
// fewer, a 4,096-tuple tile still writes runs of several tuples per bucket.
constexpr uint32_t kTwoLevelMinLog2 = 11;
// Heavy keys whose counting-pass accumulators are replicated per lane.
constexpr uint32_t kHotHeavy = 32;

__device__ __forceinline__ uint32_t find_window(const uint32_t *prefix, uint32_t n, uint32_t t) {
    // largest w with prefix[w] <= t  (prefix has n+1 entries, prefix[0] = 0)
    uint32_t lo = 0, hi = n;  // answer in [lo, hi)
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (prefix[mid] <= t) lo = mid; else hi = mid;
    }
    return lo;
}

// Partitioning model of the CTA's window: learned (when it has a model that
// did not fall back) or plain radix on the key's low bits.
// The CTA's copy of the model lives in shared memory (`core`).
struct Classifier {
    const LearnedCore *m;   // null: radix
    uint32_t mask;
    __device__ __forceinline__ uint32_t bucket(uint32_t key) const {
        return m ? learned_bucket(*m, key) : (key & mask);
    }
};

// The window's model in global memory, or null for radix partitioning.
__device__ __forceinline__ const LearnedModel *model_of(const WinPlan &wp, const LearnedModel *models) {
    return (wp.model != 0xFFFFFFFFu && !models[wp.model].fallback) ? &models[wp.model] : nullptr;
}

// ---- compacted windows joined from sorted tiles
// The light tuples of a compacted learned window are few, so they need not be
// counted, scanned and scattered: each tile of the compact array is sorted by
// bucket in place (part_light_kernel) and the join takes a bucket's runs out of
// all tiles (rows_join).  z = 1.5, 8 x 2^24 (6.4 M light tuples): counting,
// scan, scatter and join took 160 us, sorting and join 109.  (Sorting every
// tile of the other windows while they are counted, with rows of 512 to 2,048
// buckets, lost: runs of one to four tuples, 2 x 5 M at z = 1.0 668 us against
// 541, 1 M 232 against 218.)
constexpr uint32_t kRowsTilesMax = 2560;      // compact tiles of a window's two sides in a bucket's row list
constexpr uint32_t kRowsMaxLog2 = 9;          // more buckets: runs of a few tuples per tile

// Whether window w takes this form.  ccnt: the compacted light tuples per
// window side, once the counting pass is done.
__device__ __forceinline__ bool rows_form(const WinPlan &wp, uint32_t w, const LearnedModel *models,
                                          const uint32_t *ccnt) {
    if (!wp.rows || wp.model == 0xFFFFFFFFu) return false;
    const LearnedModel &m = models[wp.model];
    if (m.fallback || !m.n_heavy || !m.compact || m.log2_buckets > kRowsMaxLog2) return false;
    const uint32_t tiles = (ccnt[2 * w] + kTile - 1) / kTile + (ccnt[2 * w + 1] + kTile - 1) / kTile;
    return tiles <= kRowsTilesMax;
}

// All threads of the CTA; ends with a barrier when the window has a model.
__device__ __forceinline__ Classifier make_classifier(const WinPlan &wp, const LearnedModel *gm, LearnedCore &core) {
    Classifier c;
    c.m = nullptr;
    c.mask = (1u << wp.log2_buckets) - 1u;
    if (gm) {
        copy_to_smem(&core, gm, sizeof(LearnedCore));
        c.m = &core;
    }
    return c;
}

// ------------------------------------------------------------------ 1. histogram
// Also aggregates heavy keys of learned windows: per heavy key, count and
// sum of fr (left) / gs (right); heavy tuples are not partitioned.
__global__ void __launch_bounds__(kPartThreads, 2)
part_hist_kernel(const sjbg_tuple *__restrict__ L, const sjbg_tuple *__restrict__ R, const WinPlan *__restrict__ wins,
                 uint32_t nwin, const uint32_t *__restrict__ tileL, const uint32_t *__restrict__ tileR,
                 const uint32_t *__restrict__ hgroupL, const uint32_t *__restrict__ hgroupR,
                 uint32_t *__restrict__ cnt, uint32_t B, const LearnedModel *__restrict__ models,
                 HeavyAcc *__restrict__ hacc, uint64_t *__restrict__ compL, uint64_t *__restrict__ compR,
                 uint32_t *__restrict__ ccnt, uint32_t *__restrict__ rows) {
    extern __shared__ __align__(16) uint32_t hist[];   // P counters, then (coarse output) the tile stage
    __shared__ HeavySet hs;
    // heavy-key sums as two 32-bit words: native 32-bit shared atomics, with
    // the low word's carry (seen in its returned old value) added to the high
    // word.  The kHotHeavy heaviest keys (ids 0 .. kHotHeavy-1, heaviest first)
    // have one copy per lane after the kMaxHeavy shared ones: copy kMaxHeavy +
    // 32 * id + lane sits in the lane's own bank, so the many lanes of a warp
    // that hold the same hot key update it without bank conflicts.
    constexpr uint32_t kHeavySlotsAcc = kMaxHeavy + 32 * kHotHeavy;
    __shared__ uint32_t hcnt[kHeavySlotsAcc], hsum_lo[kHeavySlotsAcc], hsum_hi[kHeavySlotsAcc];
    // this CTA covers an equal share of one window side's tiles: the side has
    // hgroup[w + 1] - hgroup[w] counting CTAs ("hist groups")
    const bool right = blockIdx.x >= hgroupL[nwin];
    const uint32_t g = right ? blockIdx.x - hgroupL[nwin] : blockIdx.x;
    const uint32_t *hp = right ? hgroupR : hgroupL;
    const uint32_t *tp = right ? tileR : tileL;
    const uint32_t w = find_window(hp, nwin, g);
    const WinPlan wp = wins[w];
    __shared__ LearnedCore core;
    const LearnedModel *gm = model_of(wp, models);
    const Classifier cls = make_classifier(wp, gm, core);
    const bool heavy = cls.m && cls.m->n_heavy;
    const bool compact = heavy && cls.m->compact;
    // compact arrays: window w's side starts at its first tile * kTile
    uint64_t *cdst = compact ? (right ? compR : compL) + (uint64_t)tp[w] * kTile : nullptr;
    // coarse output (every window that is not compacted, when rows is given):
    // each tile's light tuples, sorted by coarse partition, go to the same
    // tile-sized region of the output; the tile's row holds the coarse offsets
    const bool coarse = rows != nullptr && !compact && wp.two_level;
    const uint32_t lgC = coarse_bits(wp.log2_buckets), cshift = wp.log2_buckets - lgC, ncoarse = 1u << lgC;
    __shared__ uint32_t ccnt_s[kCoarseMax], cpre_s[kCoarseMax + 1];
    uint64_t *stage = reinterpret_cast<uint64_t *>(hist + ((1u << wp.log2_buckets) + 1) / 2 * 2);
    uint64_t *coarse_out = coarse ? (right ? compR : compL) + (uint64_t)tp[w] * kTile : nullptr;
    uint32_t *rows_side = coarse ? rows + (right ? tileL[nwin] : 0) * kRow : nullptr;
    if (coarse)
        for (uint32_t i = threadIdx.x; i < ncoarse; i += blockDim.x) ccnt_s[i] = 0;
    const uint64_t nside = right ? wp.n_right : wp.n_left;
    const uint32_t side_tiles = tp[w + 1] - tp[w], ncta = hp[w + 1] - hp[w], j = g - hp[w];
    const uint32_t t_first = (uint32_t)((uint64_t)j * side_tiles / ncta);   // tile indices inside the window side
    const uint32_t t_end = (uint32_t)((uint64_t)(j + 1) * side_tiles / ncta);
    // counters of the buckets in use: the model's own fan-out when there is one
    const uint32_t P = 1u << (cls.m ? cls.m->log2_buckets : wp.log2_buckets);
    for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) hist[i] = 0;
    if (heavy) {
        for (uint32_t i = threadIdx.x; i < kHeavySlotsAcc; i += blockDim.x) { hcnt[i] = 0; hsum_lo[i] = 0; hsum_hi[i] = 0; }
        heavy_set_load(hs, gm);   // ends with a barrier
    }
    SJBG_BARRIER();
    // heavy keys are summed with shared atomics only: measured, that beats
    // keeping the hottest keys' sums in registers (fewer instructions per tuple
    // outweigh the atomics' serialisation on the hottest keys)
    constexpr int kPer = kTile / kPartThreads;
    const sjbg_tuple *base = right ? R + wp.right_off : L + wp.left_off;
    // key and val of the thread's tuples of tile tt (the sectors read are those
    // of whole tuples, the registers half)
    auto load_tile = [&](uint32_t tt, uint2 (&v)[kPer]) {
        const uint64_t start = (uint64_t)tt * kTile;
        const uint32_t n = (uint32_t)(nside - start < (uint64_t)kTile ? nside - start : (uint64_t)kTile);
        const uint2 *src = reinterpret_cast<const uint2 *>(base + start);
#pragma unroll
        for (int k = 0; k < kPer; k++) {
            const uint32_t i = threadIdx.x + k * kPartThreads;
            v[k] = i < n ? __ldg(src + 2 * i) : make_uint2(0u, 0u);
        }
    };
    // compacted windows: each warp buffers its light tuples in its share of the
    // stage (which only coarse output uses otherwise); wn is warp-uniform
    constexpr uint32_t kWarpBuf = kTile / (kPartThreads / 32);   // a warp's tile fits an empty buffer
    uint64_t *wbuf = stage + warp_id() * kWarpBuf;
    uint32_t wn = 0;
    auto flush_light = [&]() {
        uint32_t base = 0;
        if (lane_id() == 0) base = atomicAdd(&ccnt[2 * w + (right ? 1 : 0)], wn);
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        __syncwarp();   // the buffer's writes are visible to every lane
        for (uint32_t j = lane_id(); j < wn; j += 32) cdst[base + j] = wbuf[j];
        __syncwarp();   // read before it is refilled
        wn = 0;
    };
    // The counting loop, compiled once per kind of window (heavy keys, compacted
    // light tuples, coarse output, learned or radix buckets), so that none of
    // the mode tests runs per tuple.
    auto count_tiles = [&](auto heavy_t, auto compact_t, auto coarse_t, auto learned_t) {
        constexpr bool kHeavy = decltype(heavy_t)::value, kCompact = decltype(compact_t)::value;
        constexpr bool kCoarse = decltype(coarse_t)::value, kLearned = decltype(learned_t)::value;
        auto bucket_of = [&](uint32_t key) -> uint32_t {
            if constexpr (kLearned) return learned_bucket(*cls.m, key);
            else return key & cls.mask;
        };
        // software pipeline: tile tt+1 is in flight while tile tt is counted
        uint2 nv[kPer];
        if (t_first < t_end) load_tile(t_first, nv);
        for (uint32_t tt = t_first; tt < t_end; tt++) {
            const uint64_t start = (uint64_t)tt * kTile;
            const uint32_t n = (uint32_t)(nside - start < (uint64_t)kTile ? nside - start : (uint64_t)kTile);
            uint2 v[kPer];
#pragma unroll
            for (int k = 0; k < kPer; k++) v[k] = nv[k];
            if (tt + 1 < t_end) load_tile(tt + 1, nv);
            uint32_t lightmask = 0;
            uint32_t pk[kPer];   // coarse output: coarse << 16 | rank inside the tile's coarse run, or ~0u
            // the tuples of a tile, compiled apart for full tiles (no bounds test)
            auto count_tuples = [&](auto full_t) {
            constexpr bool kFull = decltype(full_t)::value;
            auto lookup = [&](int k) {
                return kFull || threadIdx.x + k * kPartThreads < n ? heavy_find(hs, v[k].x) : kHeavyBucket;
            };
            // the next tuple's lookup is under way while one is summed, and the count
            // is added while the low word's old value returns (2 x 2^24: z = 1.0
            // 1,175 -> 1,123 us; four lookups, then four sums: z = 1.5 406 -> 431)
            uint32_t next_hid = kHeavyBucket;
            if constexpr (kHeavy) next_hid = lookup(0);
#pragma unroll
            for (int k = 0; k < kPer; k++) {
                const uint32_t i = threadIdx.x + k * kPartThreads;
                const bool valid = kFull || i < n;
                const uint32_t key = v[k].x, val = v[k].y;
                pk[k] = 0xFFFFFFFFu;
                if constexpr (kHeavy) {
                    const uint32_t hid = next_hid;
                    if (k + 1 < kPer) next_hid = lookup(k + 1);
                    if (hid != kHeavyBucket) {
                        const unsigned long long f = sjbg_fside(val, right ? 1u : 0u);   // one mix, either side
                        const uint32_t a = hid < kHotHeavy ? kMaxHeavy + 32u * hid + lane_id() : hid;
                        const uint32_t flo = (uint32_t)f;
                        const uint32_t old = atomicAdd(&hsum_lo[a], flo);
                        atomicAdd(&hcnt[a], 1u);
                        atomicAdd(&hsum_hi[a], add_carry((uint32_t)(f >> 32), old, flo));
                    } else if (valid) {
                        // light keys: compacted windows count or sort them in part_light
                        if constexpr (kCompact) {
                            lightmask |= 1u << k;
                        } else {
                            const uint32_t b = bucket_of(key);
                            atomicAdd(&hist[b], 1u);
                            if constexpr (kCoarse) pk[k] = ((b >> cshift) << 16) | atomicAdd(&ccnt_s[b >> cshift], 1u);
                        }
                    }
                } else {
                    // plain partitioning: one shared atomic per tuple (measured faster
                    // than combining a warp's equal buckets first, skewed keys included)
                    const uint32_t b = valid ? bucket_of(key) : 0u;
                    if (valid) atomicAdd(&hist[b], 1u);
                    if constexpr (kCoarse)
                        if (valid) pk[k] = ((b >> cshift) << 16) | atomicAdd(&ccnt_s[b >> cshift], 1u);
                }
            }
            };
            if (n == (uint32_t)kTile) count_tuples(std::true_type{});
            else count_tuples(std::false_type{});
            if constexpr (kCoarse) {
                SJBG_BARRIER();   // every rank of the tile is assigned
                uint32_t *row = rows_side + (uint64_t)(tp[w] + tt) * kRow;
                if (warp_id() == 0) {
                    // exclusive offsets of the (at most 128) coarse runs; counters reset for the next tile
                    uint32_t a[kCoarseMax / 32], sum = 0;
#pragma unroll
                    for (int q = 0; q < (int)(kCoarseMax / 32); q++) {
                        const uint32_t c = lane_id() * (kCoarseMax / 32) + q;
                        a[q] = c < ncoarse ? ccnt_s[c] : 0u;
                        sum += a[q];
                    }
                    uint32_t tot;
                    uint32_t run = warp_excl_scan(sum, &tot);
#pragma unroll
                    for (int q = 0; q < (int)(kCoarseMax / 32); q++) {
                        const uint32_t c = lane_id() * (kCoarseMax / 32) + q;
                        if (c < ncoarse) {
                            cpre_s[c] = run;
                            row[c] = run;
                            ccnt_s[c] = 0;
                        }
                        run += a[q];
                    }
                    if (lane_id() == 0) {
                        cpre_s[ncoarse] = tot;
                        row[ncoarse] = tot;
                    }
                }
                SJBG_BARRIER();
#pragma unroll
                for (int k = 0; k < kPer; k++)
                    if (pk[k] != 0xFFFFFFFFu)
                        stage[cpre_s[pk[k] >> 16] + (pk[k] & 0xFFFFu)] = ((uint64_t)v[k].y << 32) | v[k].x;
                SJBG_BARRIER();
                // the tile's light tuples, contiguous per coarse run, written out whole
                const uint32_t nl = cpre_s[ncoarse];
                uint64_t *dst = coarse_out + (uint64_t)tt * kTile;
                for (uint32_t i = threadIdx.x; i < nl; i += blockDim.x) dst[i] = stage[i];
            }
            if constexpr (kCompact) {
                // the tile's light tuples go to the warp's buffer as (key,val) words
                // (warp scan, no block barrier); a full buffer is written out to the
                // window side's compact array with one global reservation
                const uint32_t nl = __popc(lightmask);
                uint32_t wt;
                const uint32_t ex = warp_excl_scan(nl, &wt);
                if (wn + wt > kWarpBuf) flush_light();
                uint32_t pos = wn + ex;
#pragma unroll
                for (int k = 0; k < kPer; k++)
                    if ((lightmask >> k) & 1u) wbuf[pos++] = ((uint64_t)v[k].y << 32) | v[k].x;
                wn += wt;
            }
        }
        if constexpr (kCompact)
            if (wn) flush_light();
    };
    using T = std::true_type;
    using F = std::false_type;
    if (compact) count_tiles(T{}, T{}, F{}, T{});
    else if (heavy && coarse) count_tiles(T{}, F{}, T{}, T{});
    else if (heavy) count_tiles(T{}, F{}, F{}, T{});
    else if (cls.m && coarse) count_tiles(F{}, F{}, T{}, T{});
    else if (cls.m) count_tiles(F{}, F{}, F{}, T{});
    else if (coarse) count_tiles(F{}, F{}, T{}, F{});
    else count_tiles(F{}, F{}, F{}, F{});
    SJBG_BARRIER();
    uint32_t *dst = cnt + (right ? B : 0) + wp.bucket_base;
    for (uint32_t i = threadIdx.x; i < P; i += blockDim.x)
        if (hist[i]) atomicAdd(&dst[i], hist[i]);
    if (heavy) {
        // fold the hot keys' per-lane copies into their shared slots: warp q sums key q's
        for (uint32_t q = warp_id(); q < kHotHeavy; q += blockDim.x >> 5) {
            const uint32_t a = kMaxHeavy + 32u * q + lane_id();
            uint32_t c = hcnt[a];
            unsigned long long sm = ((unsigned long long)hsum_hi[a] << 32) | hsum_lo[a];
            sm = warp_sum_u64(sm);
            for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xFFFFFFFFu, c, o);
            if (lane_id() == 0) {
                // slot q itself is never updated by the counting loop
                hcnt[q] = c;
                hsum_lo[q] = (uint32_t)sm;
                hsum_hi[q] = (uint32_t)(sm >> 32);
            }
        }
        SJBG_BARRIER();
        HeavyAcc *ha = hacc + (uint64_t)w * kMaxHeavy;
        for (uint32_t i = threadIdx.x; i < cls.m->n_heavy; i += blockDim.x) {
            if (!hcnt[i]) continue;
            const unsigned long long sm = ((unsigned long long)hsum_hi[i] << 32) | hsum_lo[i];
            if (right) {
                atomicAdd(&ha[i].cnt_r, (unsigned long long)hcnt[i]);
                atomicAdd(&ha[i].sum_r, sm);
            } else {
                atomicAdd(&ha[i].cnt_l, (unsigned long long)hcnt[i]);
                atomicAdd(&ha[i].sum_l, sm);
            }
        }
    }
}

// Per window side, the tiles (or fine items, or buckets) that each later pass
// has work for, as exclusive prefixes over the windows, written once the
// counting pass is done: kind 0 part_light (the compacted windows' light
// tiles), kind 1 part_scatter (those, plus every tile of a single-level window
// that was not compacted), kind 2 part_fine (two-level windows that were not
// compacted), kind 3 part_light too (the light tiles of compacted windows joined
// from sorted tiles, which the others leave out), kind 4 rows_join (buckets of
// windows joined from sorted tiles; left array only).
// Array 2 * kind + side (left 0, right 1) of n + 1 entries.  One warp per array.
enum : uint32_t { kWorkLight = 0, kWorkScatter = 1, kWorkFine = 2, kWorkSort = 3, kWorkRows = 4, kWorkArrays = 9 };
__global__ void part_work_kernel(const WinPlan *__restrict__ wins, uint32_t nwin, const uint32_t *__restrict__ tileL,
                                 const uint32_t *__restrict__ tileR, const uint32_t *__restrict__ itemL,
                                 const uint32_t *__restrict__ itemR, const LearnedModel *__restrict__ models,
                                 const uint32_t *__restrict__ ccnt, uint32_t *__restrict__ work) {
    const uint32_t a = warp_id();
    if (a >= kWorkArrays) return;   // whole warp
    const uint32_t kind = a >> 1, right = a & 1u;
    const uint32_t *tp = right ? tileR : tileL, *ip = right ? itemR : itemL;
    uint32_t *out = work + a * (nwin + 1);
    uint32_t carry = 0;
    for (uint32_t base = 0; base < nwin; base += 32) {
        const uint32_t w = base + lane_id();
        uint32_t c = 0;
        if (w < nwin) {
            const WinPlan wp = wins[w];
            const LearnedModel *gm = model_of(wp, models);
            const bool compact = gm && gm->n_heavy && gm->compact;
            const uint32_t light = (ccnt[2 * w + right] + kTile - 1) / kTile;
            const bool form = rows_form(wp, w, models, ccnt);
            if (kind == kWorkRows) c = form ? 1u << gm->log2_buckets : 0u;
            else if (kind == kWorkSort) c = form ? light : 0u;
            else if (form) c = 0;
            else if (kind == kWorkLight) c = compact ? light : 0u;
            else if (kind == kWorkScatter) c = compact ? light : (wp.two_level ? 0u : tp[w + 1] - tp[w]);
            else c = (wp.two_level && !compact) ? ip[w + 1] - ip[w] : 0u;
        }
        uint32_t tot;
        const uint32_t ex = warp_excl_scan(c, &tot);
        if (w < nwin) out[w] = carry + ex;
        carry += tot;
    }
    if (lane_id() == 0) out[nwin] = carry;
}

// Work item t of a persistent pass over prefix arrays pl (left) / pr (right):
// its window side and the index of the item inside the window side.
struct WorkItem {
    uint32_t w, local;
    bool right;
};
__device__ __forceinline__ WorkItem work_item(const uint32_t *pl, const uint32_t *pr, uint32_t nwin, uint32_t t) {
    WorkItem it;
    it.right = t >= pl[nwin];
    const uint32_t *p = it.right ? pr : pl;
    const uint32_t x = it.right ? t - pl[nwin] : t;
    it.w = find_window(p, nwin, x);
    it.local = x - p[it.w];
    return it;
}

// The compacted light tuples of compacted learned windows (part_hist only wrote
// them out).  Work kind 0: bucket counts, for the scatter.  Work kind 3: a tile
// of a window joined from sorted tiles is sorted by bucket (in place: it is in
// registers before it is written) and gets its row.  Persistent CTAs over both.
__global__ void __launch_bounds__(kPartThreads, 2)
part_light_kernel(const WinPlan *__restrict__ wins, uint32_t nwin, const uint32_t *__restrict__ tileL,
                  const uint32_t *__restrict__ tileR, const uint32_t *__restrict__ work, uint32_t *__restrict__ counts,
                  uint32_t B, const LearnedModel *__restrict__ models, uint64_t *__restrict__ compL,
                  uint64_t *__restrict__ compR, const uint32_t *__restrict__ ccnt, uint16_t *__restrict__ rows16,
                  uint32_t rstride) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ LearnedCore core;
    __shared__ uint32_t warp_tot[32];
    uint64_t *stage = reinterpret_cast<uint64_t *>(smem_raw);
    uint32_t *cnt = reinterpret_cast<uint32_t *>(stage + kTile);
    const uint32_t *cl = work + 2 * kWorkLight * (nwin + 1), *cr = cl + (nwin + 1);
    const uint32_t *pl = work + 2 * kWorkSort * (nwin + 1), *pr = pl + (nwin + 1);
    const uint32_t counted = cl[nwin] + cr[nwin], items = counted + pl[nwin] + pr[nwin];
    uint32_t cur = 0xFFFFFFFFu;   // window of the model in core
    for (uint32_t bt = blockIdx.x; bt < items; bt += gridDim.x) {
        const bool sort = bt >= counted;
        const WorkItem it = sort ? work_item(pl, pr, nwin, bt - counted) : work_item(cl, cr, nwin, bt);
        const uint32_t side_tile = (it.right ? tileR : tileL)[it.w] + it.local;
        uint64_t *words = (it.right ? compR : compL) + (uint64_t)side_tile * kTile;
        const uint32_t left = ccnt[2 * it.w + (it.right ? 1 : 0)] - it.local * kTile, n = min((uint32_t)kTile, left);
        uint64_t e[kTile / kPartThreads];
#pragma unroll
        for (int k = 0; k < kTile / kPartThreads; k++) {
            const uint32_t i = threadIdx.x + k * kPartThreads;
            e[k] = i < n ? words[i] : 0ull;
        }
        SJBG_BARRIER();   // the previous tile's readers of the stage, its counters and its model are done
        if (it.w != cur) copy_to_smem(&core, &models[wins[it.w].model], sizeof(LearnedCore));   // ends with a barrier
        cur = it.w;
        const uint32_t P = 1u << core.log2_buckets;
        for (uint32_t i = threadIdx.x; i < P; i += kPartThreads) cnt[i] = 0;
        SJBG_BARRIER();
        uint32_t br[kTile / kPartThreads];   // bucket << 16 | rank
#pragma unroll
        for (int k = 0; k < kTile / kPartThreads; k++)
            if (threadIdx.x + k * kPartThreads < n) {
                const uint32_t b = learned_bucket(core, (uint32_t)e[k]);
                br[k] = (b << 16) | atomicAdd(&cnt[b], 1u);
            }
        SJBG_BARRIER();
        if (!sort) {
            uint32_t *dst = counts + (it.right ? B : 0) + wins[it.w].bucket_base;
            for (uint32_t i = threadIdx.x; i < P; i += kPartThreads)
                if (cnt[i]) atomicAdd(&dst[i], cnt[i]);
            continue;
        }
        tile_scan(cnt, P, warp_tot);
#pragma unroll
        for (int k = 0; k < kTile / kPartThreads; k++)
            if (threadIdx.x + k * kPartThreads < n) stage[cnt[br[k] >> 16] + (br[k] & 0xFFFFu)] = e[k];
        uint16_t *row = rows16 + ((uint64_t)(it.right ? tileL[nwin] : 0) + side_tile) * rstride;
        for (uint32_t i = threadIdx.x; i < P; i += kPartThreads) row[i] = (uint16_t)cnt[i];
        if (threadIdx.x == 0) row[P] = (uint16_t)n;
        SJBG_BARRIER();
        for (uint32_t i = threadIdx.x; i < n; i += kPartThreads) words[i] = stage[i];
    }
}

// Heavy keys' contribution per window: count += |L_k||R_k|, prod += (sum fr)(sum gs).
__global__ void heavy_finish_kernel(const WinPlan *__restrict__ wins, uint32_t nwin,
                                    const LearnedModel *__restrict__ models, const HeavyAcc *__restrict__ hacc,
                                    WinAcc *__restrict__ acc) {
    const uint32_t w = blockIdx.x;
    const WinPlan wp = wins[w];
    if (wp.model == 0xFFFFFFFFu) return;
    if (models[wp.model].fallback) {   // 1: the model overflowed; 2: radix chosen by cost
        if (threadIdx.x == 0) acc[w].info = models[wp.model].fallback == 2u ? kInfoRadixByCost : kInfoFallback;
        return;
    }
    const uint32_t nh = models[wp.model].n_heavy;
    if (threadIdx.x == 0) acc[w].info = kInfoLearned | ((unsigned long long)nh << 32);
    unsigned long long c = 0, p = 0;
    for (uint32_t i = threadIdx.x; i < nh; i += blockDim.x) {
        const HeavyAcc a = hacc[(uint64_t)w * kMaxHeavy + i];
        c += a.cnt_l * a.cnt_r;
        p += a.sum_l * a.sum_r;
    }
    flush_acc(&acc[w], c, 0, p);
}

// ------------------------------------------------------------------ 2. scan
// Single-CTA exclusive scan of the bucket counts -> start and cursor.  The
// left side (counts [0, B)) and the right side (counts [B, 2B)) are scanned
// separately: each side's offsets index its own partitioned array.
__global__ void __launch_bounds__(1024) part_scan_kernel(const uint32_t *__restrict__ cnt, uint32_t *__restrict__ start,
                                                         uint32_t *__restrict__ cursor, uint32_t B) {
    __shared__ uint32_t warp_tot[32];
    __shared__ uint32_t carry_s;
    constexpr uint32_t kItems = 4;
    const uint32_t chunk = blockDim.x * kItems;
    for (uint32_t side = 0; side < 2; side++) {
        const uint32_t lo = side * B, hi = lo + B;
        if (threadIdx.x == 0) carry_s = 0;
        SJBG_BARRIER();
        for (uint32_t base = lo; base < hi; base += chunk) {
            uint32_t v[kItems], s = 0;
#pragma unroll
            for (uint32_t k = 0; k < kItems; k++) {
                const uint32_t i = base + threadIdx.x * kItems + k;
                v[k] = i < hi ? cnt[i] : 0;
                s += v[k];
            }
            uint32_t wt;
            const uint32_t ex = warp_excl_scan(s, &wt);
            if (lane_id() == 31) warp_tot[warp_id()] = ex + s;
            SJBG_BARRIER();
            if (warp_id() == 0) {
                const uint32_t x = lane_id() < (blockDim.x >> 5) ? warp_tot[lane_id()] : 0;
                uint32_t tt;
                warp_tot[lane_id()] = warp_excl_scan(x, &tt);
            }
            SJBG_BARRIER();
            uint32_t run = carry_s + warp_tot[warp_id()] + ex;
#pragma unroll
            for (uint32_t k = 0; k < kItems; k++) {
                const uint32_t i = base + threadIdx.x * kItems + k;
                if (i < hi) {
                    start[i] = run;
                    cursor[i] = run;
                }
                run += v[k];
            }
            SJBG_BARRIER();
            if (threadIdx.x == blockDim.x - 1) carry_s = run;
            SJBG_BARRIER();
        }
    }
}

// One piece of the join list with what its join reads before the tuples: a
// bucket's build run and (a piece of) its probe run, their sides, the window
// and its radix bits.
struct __align__(16) JoinItem {
    uint32_t nB, nP, sB, sP;   // tuples and first position of the build run and of the probe piece
    uint32_t w, lg, flags, pad;   // window; low key bits that all keys of the bucket share; kItem*
};
static_assert(sizeof(JoinItem) == 32, "two 16-byte words per join item");
enum : uint32_t {
    kItemModel = 1u,    // a learned bucket: a key range rather than a residue class
    kItemSwap = 2u,     // built from the right side, probed by the left
    kItemRaw = 4u,      // an unpartitioned window: positions index its sides' tuples
    kItemHot = 8u       // a piece of a build run longer than its table
};

// A bucket's pieces: nb build pieces times np probe pieces, every pair of them
// one item (count and checksum are sums over the pairs).
struct JoinGrid {
    uint32_t nb, np;
    __host__ __device__ uint32_t items() const { return nb * np; }
};

// A bucket is cut into pieces of about `chunk` probe tuples, joined by
// different CTAs; each builds the bucket's table again, so a piece has at least
// as many probes as the build run.  A longer build run (cap: a table's slots)
// is a hot key's or a low fan-out's: up to kHotRuns tables long it is joined in
// one piece, whose refused keys are compacted in place (only one CTA may do
// that); beyond, both runs are cut, into at most kHotSplit pieces each, or one
// CTA would join millions of tuples alone (8 x 2^24, z = 1.5, one hot key in
// the buckets: 6.1 ms).  With s pieces of each run a bucket costs s times its
// tuples, spread over s^2 CTAs: s is the root of kHotFactor times the CTAs'
// number times the bucket's share of the call's tuples (its tuples / hot_unit); at
// a factor of 1 and with equal hot buckets one piece takes as long as an even
// share of all of them, and buckets differ.  Whole calls, s = 16 / factor 1 / 2 /
// 4 / one piece: 32 windows of 2^20, z = 1.25 1.59 / 1.55 / 1.32 / 1.29 / 1.43 ms,
// z = 1.5 2.46 / 1.58 / 1.49 / 1.53 / 1.80; one of 2^22, z = 1.5 708 / 542 / 534 /
// 580 / 2,590 us; 128 of 2^18, z = 1.5 1.30 / 1.28 / 1.25 / 1.16 / 1.19 ms.
constexpr uint32_t kHotRuns = 8, kHotSplit = 16, kHotFactor = 4;
__device__ __forceinline__ JoinGrid join_grid(uint32_t nB, uint32_t nP, uint32_t chunk, uint32_t cap, uint32_t hot_unit) {
    JoinGrid g{1, 1};
    if (nB < cap) {
        const uint32_t per = chunk > nB ? chunk : nB;
        g.np = (uint32_t)(((uint64_t)nP + per / 2) / per);   // rounded: a piece is at most 1.5 chunks
        if (g.np == 0) g.np = 1;
    } else if (nB > kHotRuns * cap && nP > kHotRuns * cap) {
        const uint32_t per = kHotRuns / 2 * cap, kb = nB / per, kp = nP / per;   // at least 2 of each
        const uint32_t s = min(kHotSplit, max(1u, (uint32_t)(sqrtf(((float)nB + (float)nP) / (float)hot_unit) + 0.5f)));
        g.nb = min(kb, s);
        g.np = min(kp, s);
    }
    return g;
}

// The most items a call can have: one per bucket and, by join_grid, at most one
// more per chunk of probes and kHotSplit more per kHotRuns / 2 tables of a side.
static inline uint64_t join_items_bound(uint64_t buckets, uint64_t tuples, uint32_t chunk, uint32_t cap) {
    return buckets + tuples / chunk + tuples / (kHotRuns / 2 * cap) * kHotSplit;
}

// Item q of a bucket: its build piece and its probe piece.
__device__ __forceinline__ void item_piece(JoinItem &ji, const JoinGrid &g, uint32_t q, uint32_t nB, uint32_t sB,
                                           uint32_t nP, uint32_t sP) {
    const uint32_t ib = q / g.np, ip = q - ib * g.np;
    const uint32_t b0 = (uint32_t)((uint64_t)nB * ib / g.nb), p0 = (uint32_t)((uint64_t)nP * ip / g.np);
    ji.sB = sB + b0;
    ji.nB = (uint32_t)((uint64_t)nB * (ib + 1) / g.nb) - b0;
    ji.sP = sP + p0;
    ji.nP = (uint32_t)((uint64_t)nP * (ip + 1) / g.np) - p0;
}

// Whether a window needs no partitioning: its smaller side is one bucket, so
// the join reads the tuples themselves.  Sides differ much in real batches (an
// idle stream against a busy one), and partitioning the larger side into one
// bucket would copy it for nothing.  With the fan-out by the smaller side, the
// smaller side built and long runs cut, the bucket joins of the 1,024 windows
// above went from 6.60 to 4.17 ms, their counting from 0.70 to 0.57 and their
// scatter from 1.75 to 1.35.
__host__ __device__ __forceinline__ bool raw_window(const WinPlan &wp) { return wp.raw != 0; }

// Per window, one CTA: exclusive scan of the window's bucket counts on each
// side, starting at the window's base in that side's partitioned array (the
// tuples of the windows before it: baseL / baseR), giving the bucket starts
// and scatter cursors; then every bucket with tuples on both sides is appended
// to the join list (items, length *jn: nothing else can match), in pieces.
// either: the join may build from either side, and builds from the smaller;
// otherwise it builds from the left.
constexpr uint32_t kScanOwn = 4;
__global__ void __launch_bounds__(1024)
part_scan_win_kernel(const WinPlan *__restrict__ wins, const uint32_t *__restrict__ baseL,
                     const uint32_t *__restrict__ baseR, const uint32_t *__restrict__ cnt,
                     uint32_t *__restrict__ start, uint32_t *__restrict__ cursor, uint32_t B,
                     const LearnedModel *__restrict__ models, JoinItem *__restrict__ items,
                     uint32_t *__restrict__ jn, uint32_t chunk, uint32_t cap, uint32_t hot_unit, bool either,
                     const uint32_t *__restrict__ ccnt) {
    __shared__ uint32_t warp_tot[32];
    __shared__ uint32_t carry_s;
    const uint32_t w = blockIdx.x;
    const WinPlan wp = wins[w];
    if (raw_window(wp)) {   // its pieces, straight over the tuples
        const uint32_t nL = (uint32_t)wp.n_left, nR = (uint32_t)wp.n_right;
        const bool swap = either && nR < nL;
        const uint32_t nB = swap ? nR : nL, nP = swap ? nL : nR;
        const JoinGrid g = join_grid(nB, nP, chunk, cap, hot_unit);   // (the build side is below cap)
        const uint32_t k = g.items();
        if (threadIdx.x == 0) carry_s = atomicAdd(jn, k);
        SJBG_BARRIER();
        for (uint32_t i = threadIdx.x; i < k; i += blockDim.x) {
            JoinItem ji;
            item_piece(ji, g, i, nB, 0u, nP, 0u);
            ji.w = w; ji.lg = 0; ji.flags = kItemRaw | (swap ? kItemSwap : 0u); ji.pad = 0;
            items[carry_s + i] = ji;
        }
        return;
    }
    if (models && rows_form(wp, w, models, ccnt)) return;   // (whole CTA: nothing of it is in the join list)
    const uint32_t P = 1u << wp.log2_buckets, b0 = wp.bucket_base;
    constexpr uint32_t kItems = 4;
    const uint32_t tchunk = blockDim.x * kItems;
    for (uint32_t side = 0; side < 2; side++) {
        const uint32_t lo = side * B + b0, hi = lo + P;
        if (threadIdx.x == 0) carry_s = side ? baseR[w] : baseL[w];
        SJBG_BARRIER();
        for (uint32_t base = lo; base < hi; base += tchunk) {
            uint32_t v[kItems], s = 0;
#pragma unroll
            for (uint32_t k = 0; k < kItems; k++) {
                const uint32_t i = base + threadIdx.x * kItems + k;
                v[k] = i < hi ? cnt[i] : 0;
                s += v[k];
            }
            uint32_t wt;
            const uint32_t ex = warp_excl_scan(s, &wt);
            if (lane_id() == 31) warp_tot[warp_id()] = ex + s;
            SJBG_BARRIER();
            if (warp_id() == 0) {
                const uint32_t x = lane_id() < (blockDim.x >> 5) ? warp_tot[lane_id()] : 0;
                uint32_t tt;
                warp_tot[lane_id()] = warp_excl_scan(x, &tt);
            }
            SJBG_BARRIER();
            uint32_t run = carry_s + warp_tot[warp_id()] + ex;
#pragma unroll
            for (uint32_t k = 0; k < kItems; k++) {
                const uint32_t i = base + threadIdx.x * kItems + k;
                if (i < hi) {
                    start[i] = run;
                    cursor[i] = run;
                }
                run += v[k];
            }
            SJBG_BARRIER();
            if (threadIdx.x == blockDim.x - 1) carry_s = run;
            SJBG_BARRIER();
        }
    }
    // join list: one reservation per warp of joinable buckets (the starts were
    // written by this CTA, before the scan's last barrier)
    const bool model = models && model_of(wp, models) != nullptr;
    for (uint32_t i0 = 0; i0 < P; i0 += blockDim.x) {
        const uint32_t i = i0 + threadIdx.x, b = b0 + i;
        const uint32_t nL = i < P ? cnt[b] : 0u, nR = i < P ? cnt[B + b] : 0u;
        const bool swap = either && nR < nL;
        const uint32_t nB = swap ? nR : nL, nP = swap ? nL : nR;
        const JoinGrid g = join_grid(nB, nP, chunk, cap, hot_unit);
        const uint32_t k = (nL != 0u && nR != 0u) ? g.items() : 0u;
        uint32_t tot;
        const uint32_t ex = warp_excl_scan(k, &tot);
        uint32_t wbase = 0;
        if (lane_id() == 0 && tot) wbase = atomicAdd(jn, tot);
        wbase = __shfl_sync(0xFFFFFFFFu, wbase, 0) + ex;
        const uint32_t sB = k ? start[swap ? B + b : b] : 0u, sP = k ? start[swap ? b : B + b] : 0u;
        JoinItem ji;
        ji.w = w; ji.lg = wp.log2_buckets; ji.pad = 0;
        ji.flags = (model ? kItemModel : 0u) | (swap ? kItemSwap : 0u) | (g.nb > 1 ? kItemHot : 0u);
        if (k <= kScanOwn)
            for (uint32_t q = 0; q < k; q++) {
                item_piece(ji, g, q, nB, sB, nP, sP);
                items[wbase + q] = ji;
            }
        // a bucket of many pieces: its warp writes them (by one thread the list of 32
        // windows of 2^20 took 121 us at z = 1.5)
        for (unsigned many = __ballot_sync(0xFFFFFFFFu, k > kScanOwn); many; many &= many - 1) {
            const int from = __ffs(many) - 1;
            auto of = [&](uint32_t x) { return __shfl_sync(0xFFFFFFFFu, x, from); };
            const JoinGrid og{of(g.nb), of(g.np)};
            const uint32_t onB = of(nB), osB = of(sB), onP = of(nP), osP = of(sP), obase = of(wbase);
            JoinItem o = ji;
            o.flags = of(ji.flags);
            for (uint32_t q = lane_id(); q < og.items(); q += 32) {
                item_piece(o, og, q, onB, osB, onP, osP);
                items[obase + q] = o;
            }
        }
    }
}

// Block-wide exclusive scan of P (<= 16384) shared counters in place.
__device__ void block_scan_smem(uint32_t *a, uint32_t P, uint32_t *warp_tot) {
    const uint32_t per = (P + blockDim.x - 1) / blockDim.x;
    const uint32_t b0 = min(P, threadIdx.x * per), b1 = min(P, b0 + per);
    uint32_t s = 0;
    for (uint32_t i = b0; i < b1; i++) s += a[i];
    uint32_t tot;
    uint32_t ex = warp_excl_scan(s, &tot);
    if (lane_id() == 31) warp_tot[warp_id()] = ex + s;
    SJBG_BARRIER();
    if (warp_id() == 0) {
        uint32_t x = lane_id() < (blockDim.x >> 5) ? warp_tot[lane_id()] : 0, tt;
        warp_tot[lane_id()] = warp_excl_scan(x, &tt);
    }
    SJBG_BARRIER();
    uint32_t run = warp_tot[warp_id()] + ex;
    for (uint32_t i = b0; i < b1; i++) {
        uint32_t c = a[i];
        a[i] = run;
        run += c;
    }
    SJBG_BARRIER();
}

// ------------------------------------------------------------------ 3. scatter
constexpr int kScatterPer = kTile / kPartThreads;   // tuples per thread per tile

// Where a scatter work item's tuples are: the window side's tuples, or (a
// compacted window) the light tuples the counting pass packed as 8-byte words.
struct TileIn {
    const void *p;
    uint32_t n;        // tuples in the tile
    uint32_t packed;   // 8-byte (key, val) words rather than 16-byte tuples
};

__device__ __forceinline__ TileIn tile_input(const WorkItem it, const sjbg_tuple *__restrict__ L,
                                             const sjbg_tuple *__restrict__ R, const WinPlan *__restrict__ wins,
                                             const uint32_t *__restrict__ tileL, const uint32_t *__restrict__ tileR,
                                             const LearnedModel *__restrict__ models,
                                             const uint64_t *__restrict__ compL, const uint64_t *__restrict__ compR,
                                             const uint32_t *__restrict__ ccnt) {
    const bool right = it.right;
    const uint32_t w = it.w;
    const WinPlan &wp = wins[w];
    const LearnedModel *gm = model_of(wp, models);
    const bool compact = gm && gm->n_heavy && gm->compact;
    const uint64_t nside = compact ? ccnt[2 * w + (right ? 1 : 0)] : (right ? wp.n_right : wp.n_left);
    const uint64_t start = (uint64_t)it.local * kTile;
    TileIn t;
    t.n = (uint32_t)(nside - start < (uint64_t)kTile ? nside - start : (uint64_t)kTile);
    t.packed = compact ? 1u : 0u;
    if (compact)
        t.p = (right ? compR : compL) + (uint64_t)(right ? tileR : tileL)[w] * kTile + start;
    else
        t.p = (right ? R + wp.right_off : L + wp.left_off) + start;
    return t;
}

// The thread's tuples of a tile as (val << 32 | key) words, every load in flight before any use.
__device__ __forceinline__ void tile_load(const TileIn &t, uint64_t (&e)[kScatterPer]) {
#pragma unroll
    for (int k = 0; k < kScatterPer; k++) {
        const uint32_t i = threadIdx.x + k * kPartThreads;
        if (i < t.n) {
            if (t.packed) {
                e[k] = __ldg(static_cast<const uint64_t *>(t.p) + i);
            } else {
                const uint2 v = __ldg(reinterpret_cast<const uint2 *>(static_cast<const sjbg_tuple *>(t.p) + i));
                e[k] = ((uint64_t)v.y << 32) | v.x;   // key and val only
            }
        }
    }
}

// One tile whose tuples are already in e[]: local counting sort by bucket in
// shared memory, one global reservation per non-empty bucket, contiguous
// per-bucket runs written out.  As soon as the tile is staged in shared memory
// e[] is free, so the next tile's loads (next, when given) are issued into it
// before this tile's write-out: they are in flight while it runs.
__device__ __forceinline__ void scatter_tile(const WorkItem it, const TileIn in, uint64_t (&e)[kScatterPer],
                                             const TileIn *next, const WinPlan *__restrict__ wins,
                                             uint32_t *__restrict__ cursor, uint32_t B, uint64_t *__restrict__ outL,
                                             uint64_t *__restrict__ outR, const LearnedModel *__restrict__ models) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ uint32_t warp_tot[32];
    const bool right = it.right;
    const WinPlan wp = wins[it.w];
    const LearnedModel *gm = model_of(wp, models);
    const bool compact = in.packed != 0;
    const uint32_t n = in.n;
    // a model buckets into its own (often smaller) fan-out: only those counters are touched
    const uint32_t P = 1u << (gm ? gm->log2_buckets : wp.log2_buckets);

    uint64_t *stage = reinterpret_cast<uint64_t *>(smem_raw);                  // kTile
    uint16_t *sb = reinterpret_cast<uint16_t *>(stage + kTile);                // kTile bucket ids
    uint32_t *lcnt = reinterpret_cast<uint32_t *>(sb + kTile);                 // P
    uint32_t *gbase = lcnt + P;                                                // P
    __shared__ LearnedCore core;
    const Classifier cls = make_classifier(wp, gm, core);
    const bool heavy = cls.m && cls.m->n_heavy && !compact;
    __shared__ HeavySet hs;
    __shared__ uint32_t kept_s;

    for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) lcnt[i] = 0;
    if (threadIdx.x == 0) kept_s = 0;
    if (heavy) heavy_set_load(hs, gm);
    SJBG_BARRIER();
    uint32_t bk[kScatterPer], rk[kScatterPer];
#pragma unroll
    for (int k = 0; k < kScatterPer; k++) {
        const uint32_t i = threadIdx.x + k * kPartThreads;
        bk[k] = kHeavyBucket;
        if (i < n) {
            const uint32_t key = (uint32_t)e[k];
            if (!heavy || heavy_find(hs, key) == kHeavyBucket) {
                bk[k] = cls.bucket(key);
                rk[k] = atomicAdd(&lcnt[bk[k]], 1u);
            }
        }
    }
    SJBG_BARRIER();
    // the next tile into L2 (its address is known by now), so that the register
    // loads issued once this tile is staged find it there
    if (next && threadIdx.x == 0) l2_prefetch_bulk(next->p, (size_t)next->n * (next->packed ? 8u : 16u));
    // reserve one global range per non-empty bucket
    uint32_t *gcur = cursor + (right ? B : 0) + wp.bucket_base;
    uint32_t kept = 0;
    for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) {
        const uint32_t c = lcnt[i];
        gbase[i] = c ? atomicAdd(&gcur[i], c) : 0;
        kept += c;
    }
    if (heavy) atomicAdd(&kept_s, kept);
    block_scan_smem(lcnt, P, warp_tot);   // lcnt -> local offsets (ends with a barrier)
    const uint32_t nk = heavy ? kept_s : n;
#pragma unroll
    for (int k = 0; k < kScatterPer; k++) {
        if (bk[k] != kHeavyBucket) {
            const uint32_t pos = lcnt[bk[k]] + rk[k];
            stage[pos] = e[k];
            sb[pos] = (uint16_t)bk[k];
        }
    }
    if (next) tile_load(*next, e);
    SJBG_BARRIER();
    uint64_t *out = right ? outR : outL;
    for (uint32_t j = threadIdx.x; j < nk; j += blockDim.x) {
        const uint32_t b = sb[j];
        out[gbase[b] + (j - lcnt[b])] = stage[j];
    }
}

// scatter_tile for a radix window (no model, no heavy keys, not compacted):
// a tuple's bucket is key & mask, so the staged word carries it and no bucket
// array is kept; the write-out reads one per-bucket delta (global base minus
// local offset) per tuple.
__device__ __forceinline__ void scatter_tile_radix(const WorkItem it, const TileIn in, uint64_t (&e)[kScatterPer],
                                                   const TileIn *next, const WinPlan *__restrict__ wins,
                                                   uint32_t *__restrict__ cursor, uint32_t B,
                                                   uint64_t *__restrict__ outL, uint64_t *__restrict__ outR) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ uint32_t warp_tot[32];
    const WinPlan wp = wins[it.w];
    const uint32_t mask = (1u << wp.log2_buckets) - 1u, P = mask + 1u;
    const uint32_t n = in.n;
    uint64_t *stage = reinterpret_cast<uint64_t *>(smem_raw);   // kTile
    uint32_t *lcnt = reinterpret_cast<uint32_t *>(stage + kTile);  // P
    uint32_t *delta = lcnt + P;                                  // P
    for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) lcnt[i] = 0;
    SJBG_BARRIER();
    uint32_t rk[kScatterPer];
#pragma unroll
    for (int k = 0; k < kScatterPer; k++)
        if (threadIdx.x + k * kPartThreads < n) rk[k] = atomicAdd(&lcnt[(uint32_t)e[k] & mask], 1u);
    SJBG_BARRIER();
    if (next && threadIdx.x == 0) l2_prefetch_bulk(next->p, (size_t)next->n * (next->packed ? 8u : 16u));
    // reserve one global range per non-empty bucket
    uint32_t *gcur = cursor + (it.right ? B : 0) + wp.bucket_base;
    for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) {
        const uint32_t c = lcnt[i];
        delta[i] = c ? atomicAdd(&gcur[i], c) : 0;
    }
    block_scan_smem(lcnt, P, warp_tot);   // lcnt -> local offsets (ends with a barrier)
#pragma unroll
    for (int k = 0; k < kScatterPer; k++)
        if (threadIdx.x + k * kPartThreads < n) stage[lcnt[(uint32_t)e[k] & mask] + rk[k]] = e[k];
    for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) delta[i] -= lcnt[i];   // (mod 2^32)
    if (next) tile_load(*next, e);
    SJBG_BARRIER();
    uint64_t *out = it.right ? outR : outL;
    for (uint32_t j = threadIdx.x; j < n; j += blockDim.x) {
        const uint64_t x = stage[j];
        out[delta[(uint32_t)x & mask] + j] = x;
    }
}

// kRadixOnly: no window of the call has a model (compiled without the general path).
template <bool kRadixOnly>
__global__ void __launch_bounds__(kPartThreads, kRadixOnly ? 3 : 2)
part_scatter_kernel(const sjbg_tuple *__restrict__ L, const sjbg_tuple *__restrict__ R, const WinPlan *__restrict__ wins,
                    uint32_t nwin, const uint32_t *__restrict__ tileL, const uint32_t *__restrict__ tileR,
                    const uint32_t *__restrict__ workL, const uint32_t *__restrict__ workR,
                    uint32_t *__restrict__ cursor, uint32_t B, uint64_t *__restrict__ outL, uint64_t *__restrict__ outR,
                    const LearnedModel *__restrict__ models, const uint64_t *__restrict__ compL,
                    const uint64_t *__restrict__ compR, const uint32_t *__restrict__ ccnt) {
    // persistent CTAs over the tiles listed by the work prefixes workL / workR
    // (a compacted window's light tiles; a single-level window's tiles), each
    // tile's loads issued while the previous tile is written out.  Without models
    // a CTA takes a run of neighbours: the prefixes are searched once per window
    // side instead of once per tile (ten loads, one after the other, with 1,024
    // windows: 1,347 -> 1,215 us).  With models tiles cost what their light
    // tuples cost, and every gridDim.x-th spreads them better (3 x 2,000,000 at
    // z = 1.0: 113 us, by runs 119).
    const uint64_t items = workL[nwin] + workR[nwin];
    uint32_t bt = kRadixOnly ? (uint32_t)(blockIdx.x * items / gridDim.x) : blockIdx.x;
    const uint32_t bt_end = kRadixOnly ? (uint32_t)((blockIdx.x + 1) * items / gridDim.x) : (uint32_t)items;
    const uint32_t step = kRadixOnly ? 1u : gridDim.x;
    if (bt >= bt_end) return;
    WorkItem it = work_item(workL, workR, nwin, bt);
    auto last_of = [&](const WorkItem &x) {   // the last tile of x's window side
        const uint32_t *p = x.right ? workR : workL;
        return p[x.w + 1] - p[x.w] - 1;
    };
    uint32_t last = kRadixOnly ? last_of(it) : 0u;
    TileIn in = tile_input(it, L, R, wins, tileL, tileR, models, compL, compR, ccnt);
    uint64_t e[kScatterPer];
    tile_load(in, e);
    for (; bt < bt_end; bt += step) {
        SJBG_BARRIER();   // the previous tile's shared-memory readers are done
        const uint32_t nb = bt + step;
        WorkItem nit = it;
        TileIn nin = in;
        if (nb < bt_end) {
            if (kRadixOnly && it.local < last) {
                nit.local++;
            } else {
                nit = work_item(workL, workR, nwin, nb);
                if (kRadixOnly) last = last_of(nit);
            }
            nin = tile_input(nit, L, R, wins, tileL, tileR, models, compL, compR, ccnt);
        }
        if (kRadixOnly || (!in.packed && !model_of(wins[it.w], models)))
            scatter_tile_radix(it, in, e, nb < bt_end ? &nin : nullptr, wins, cursor, B, outL, outR);
        else
            scatter_tile(it, in, e, nb < bt_end ? &nin : nullptr, wins, cursor, B, outL, outR, models);
        it = nit;
        in = nin;
    }
}


// ------------------------------------------------------------------ 3'. fine pass
// Two-level windows: one work item per (window side, coarse partition c,
// group of kGroupTiles tiles) gathers the tiles' runs of partition c (about
// kTile / 2^lgC tuples each, contiguous) with asynchronous 8-byte copies into
// shared memory, and scatters them into the partition's 2^(lg - lgC) fine
// buckets: a local counting sort of up to kFineChunk tuples, one global
// reservation per fine bucket, then contiguous per-bucket runs - coalesced
// writes however many buckets the window has.  Persistent CTAs take the items
// of the windows that need the pass (part_work's prefixes) in turn.
__device__ __forceinline__ void cp_async8(void *smem, const void *gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)),
                 "l"(gmem)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Up to kFineGather tuples of an item are gathered at once (all of a typical
// item's runs, one memory latency), then sorted in chunks of kFineChunk.
// (Measured: prefetching the next item's runs into L2 from here made the pass
// slower - reading that item's rows held a warp past the gather.)
constexpr uint32_t kFineGather = 2 * kFineChunk;
constexpr size_t kFineSmem = kFineGather * sizeof(uint64_t) + kFineChunk * sizeof(uint8_t);

// An item's coarse partition c and its group of tiles [t0, t0 + G).
struct FineRuns {
    uint32_t c, t0, G;
};
__device__ __forceinline__ FineRuns fine_runs(const WorkItem it, const WinPlan *__restrict__ wins,
                                              const uint32_t *__restrict__ tileL, const uint32_t *__restrict__ tileR) {
    const uint32_t *tp = it.right ? tileR : tileL;
    const uint32_t w = it.w;
    const uint32_t ntw = tp[w + 1] - tp[w];
    const uint32_t ngroups = (ntw + kGroupTiles - 1) / kGroupTiles;
    FineRuns f;
    f.c = it.local / ngroups;
    const uint32_t g = it.local % ngroups;
    f.t0 = g * kGroupTiles;
    f.G = min(kGroupTiles, ntw - f.t0);
    return f;
}

__device__ __forceinline__ void fine_item(const WorkItem it, const WinPlan *__restrict__ wins,
                                          uint32_t nwin, const uint32_t *__restrict__ tileL,
                                          const uint32_t *__restrict__ tileR, uint32_t *__restrict__ cursor, uint32_t B,
                                          uint64_t *__restrict__ outL, uint64_t *__restrict__ outR,
                                          const LearnedModel *__restrict__ models, const uint64_t *__restrict__ srcL,
                                          const uint64_t *__restrict__ srcR, const uint32_t *__restrict__ rows) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    // kFineGather gathered tuples; a chunk is staged, sorted by fine bucket, in
    // its own part of it (its tuples are in registers by then)
    uint64_t *tmp = reinterpret_cast<uint64_t *>(smem_raw);
    uint8_t *sf = reinterpret_cast<uint8_t *>(tmp + kFineGather);   // kFineChunk fine ids
    __shared__ uint32_t runoff[kGroupTiles], runpre[kGroupTiles + 1];
    __shared__ uint32_t fcnt[kCoarseMax], floc[kCoarseMax], fbase[kCoarseMax];
    __shared__ LearnedCore core;
    const bool right = it.right;
    const uint32_t *tp = right ? tileR : tileL;
    const uint32_t w = it.w;
    const WinPlan wp = wins[w];
    const LearnedModel *gm = model_of(wp, models);   // a two-level window that was not compacted
    const uint32_t lg = wp.log2_buckets, lgC = coarse_bits(lg), cshift = lg - lgC, nfine = 1u << cshift;
    const FineRuns fr_it = fine_runs(it, wins, tileL, tileR);
    const uint32_t c = fr_it.c, t0 = fr_it.t0, G = fr_it.G;
    const Classifier cls = make_classifier(wp, gm, core);   // ends with a barrier when there is a model
    const uint32_t *rows_side = rows + (right ? tileL[nwin] : 0) * kRow;
    if (warp_id() == 0) {
        // the runs of partition c in tiles t0 .. t0 + G, and their prefix
        uint32_t len[2], sum = 0;
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const uint32_t i = lane_id() * 2 + q;
            len[q] = 0;
            if (i < G) {
                const uint32_t *row = rows_side + (uint64_t)(tp[w] + t0 + i) * kRow;
                const uint32_t off = row[c];
                len[q] = row[c + 1] - off;
                runoff[i] = (t0 + i) * kTile + off;
            }
            sum += len[q];
        }
        uint32_t tot;
        uint32_t run = warp_excl_scan(sum, &tot);
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const uint32_t i = lane_id() * 2 + q;
            if (i < G) runpre[i] = run;
            run += len[q];
        }
        if (lane_id() == 0) runpre[G] = tot;
    }
    SJBG_BARRIER();
    const uint32_t T = runpre[G];
    const uint64_t *src = (right ? srcR : srcL) + (uint64_t)tp[w] * kTile;
    uint64_t *out = right ? outR : outL;
    uint32_t *gcur = cursor + (right ? B : 0) + wp.bucket_base + (c << cshift);
    constexpr int kPer = kFineChunk / kFineThreads;
    const uint32_t nwarps = blockDim.x >> 5;
    for (uint32_t gw = 0; gw < T; gw += kFineGather) {
        const uint32_t mg = min(kFineGather, T - gw);
        // gather: warp r % nwarps copies the part of run r inside [gw, gw + mg)
        for (uint32_t r = warp_id(); r < G; r += nwarps) {
            const uint32_t a = max(runpre[r], gw), b = min(runpre[r + 1], gw + mg);
            for (uint32_t x = a + lane_id(); x < b; x += 32)
                cp_async8(tmp + (x - gw), src + runoff[r] + (x - runpre[r]));
        }
        cp_async_wait_all();
        SJBG_BARRIER();
        for (uint32_t ch = 0; ch < mg; ch += kFineChunk) {
            const uint32_t m = min(kFineChunk, mg - ch);
            uint64_t *stage = tmp + ch;
            for (uint32_t f = threadIdx.x; f < nfine; f += blockDim.x) fcnt[f] = 0;
            SJBG_BARRIER();
            uint64_t e[kPer];
            uint32_t fr[kPer];
#pragma unroll
            for (int k = 0; k < kPer; k++) {
                const uint32_t j = threadIdx.x + k * kFineThreads;
                fr[k] = 0xFFFFFFFFu;
                if (j < m) {
                    e[k] = tmp[ch + j];
                    const uint32_t f = cls.bucket((uint32_t)e[k]) & (nfine - 1);
                    fr[k] = (f << 16) | atomicAdd(&fcnt[f], 1u);
                }
            }
            SJBG_BARRIER();
            // the reservations go out now and are stored after the staging, which hides their latency
            uint32_t reserved = 0;
            if (threadIdx.x < nfine && fcnt[threadIdx.x]) reserved = atomicAdd(&gcur[threadIdx.x], fcnt[threadIdx.x]);
            if (warp_id() == 0) {
                uint32_t a[kCoarseMax / 32], sum = 0;
#pragma unroll
                for (int q = 0; q < (int)(kCoarseMax / 32); q++) {
                    const uint32_t f = lane_id() * (kCoarseMax / 32) + q;
                    a[q] = f < nfine ? fcnt[f] : 0u;
                    sum += a[q];
                }
                uint32_t tot;
                uint32_t run = warp_excl_scan(sum, &tot);
#pragma unroll
                for (int q = 0; q < (int)(kCoarseMax / 32); q++) {
                    const uint32_t f = lane_id() * (kCoarseMax / 32) + q;
                    if (f < nfine) floc[f] = run;
                    run += a[q];
                }
            }
            SJBG_BARRIER();
#pragma unroll
            for (int k = 0; k < kPer; k++) {
                if (fr[k] != 0xFFFFFFFFu) {
                    const uint32_t pos = floc[fr[k] >> 16] + (fr[k] & 0xFFFFu);
                    stage[pos] = e[k];
                    sf[pos] = (uint8_t)(fr[k] >> 16);
                }
            }
            if (threadIdx.x < nfine) fbase[threadIdx.x] = reserved;
            SJBG_BARRIER();
            for (uint32_t pos = threadIdx.x; pos < m; pos += blockDim.x) {
                const uint32_t f = sf[pos];
                out[fbase[f] + (pos - floc[f])] = stage[pos];
            }
            SJBG_BARRIER();
        }
    }
}

__global__ void __launch_bounds__(kFineThreads, 4)
part_fine_kernel(const WinPlan *__restrict__ wins, uint32_t nwin, const uint32_t *__restrict__ tileL,
                 const uint32_t *__restrict__ tileR, const uint32_t *__restrict__ work, uint32_t *__restrict__ cursor,
                 uint32_t B, uint64_t *__restrict__ outL, uint64_t *__restrict__ outR,
                 const LearnedModel *__restrict__ models, const uint64_t *__restrict__ srcL,
                 const uint64_t *__restrict__ srcR, const uint32_t *__restrict__ rows) {
    const uint32_t *pl = work + 2 * kWorkFine * (nwin + 1), *pr = pl + (nwin + 1);
    const uint32_t items = pl[nwin] + pr[nwin];
    for (uint32_t bi = blockIdx.x; bi < items; bi += gridDim.x) {
        SJBG_BARRIER();   // the previous item's shared-memory readers are done
        fine_item(work_item(pl, pr, nwin, bi), wins, nwin, tileL, tileR, cursor, B, outL, outR, models, srcL, srcR,
                  rows);
    }
}

// ------------------------------------------------------------------ 4. bucket join
constexpr uint32_t kMaxProbe = 64;   // linear-probe bound of the count tables that may fill up

// Count-table slots for buckets of about `target` left tuples (load <= 0.77).
static inline uint32_t count_table_cap(uint32_t target) { return (target * 13u / 10u + 31u) & ~31u; }

struct CountTable {
    uint32_t *keys;              // C + 1 (slot C reserved for key 0xFFFFFFFF)
    uint32_t *cnt;               // C + 1
    unsigned long long *sumf;    // C + 1
    uint32_t C;                  // slots (any size: the hash is scaled, not masked)
    uint32_t max_probe;          // kMaxProbe, or C where every key of a shorter build run has to fit (its pieces share it)
};

// Home slot of a key in a table of C slots: a 32-bit multiplicative hash scaled to [0, C).
__device__ __forceinline__ uint32_t ct_home(uint32_t key, uint32_t C) {
    return (uint32_t)(((uint64_t)slot_hash(key, 32) * C) >> 32);
}

// Insert `c` tuples of `key` with hash sum `f`.  A key that finds neither itself
// nor a free slot within max_probe slots is refused (false) and joined in a
// later pass; lookups use the same bound, so a refused key is never half-found.
// Every lane inserts its own tuple: with the sums' native 32-bit atomics this
// beats combining a warp's equal keys first, at every skew measured.
__device__ __forceinline__ bool ct_insert(const CountTable &t, uint32_t key, uint32_t c, unsigned long long f) {
    const uint32_t C = t.C;
    if (key == kEmptyKey) {
        atomicAdd(&t.cnt[C], c);
        ct_add_sum(&t.sumf[C], f);
        return true;
    }
    uint32_t s = ct_home(key, C);
    auto step = [&]() {   // the key is in slot s now
        uint32_t k = *(volatile uint32_t *)&t.keys[s];
        if (k == kEmptyKey) {
            const uint32_t prev = atomicCAS(&t.keys[s], kEmptyKey, key);
            k = prev == kEmptyKey ? key : prev;
        }
        if (k != key) {
            s = s + 1 == C ? 0 : s + 1;
            return false;
        }
        atomicAdd(&t.cnt[s], c);
        ct_add_sum(&t.sumf[s], f);
        return true;
    };
    // (a constant bound, unrolled, and the rest apart: with the bound in a register
    // the joins of 2 x 2^24 tuples at 2^10 buckets took 4.9 ms instead of 3.5)
    for (uint32_t probe = 0; probe < kMaxProbe; probe++)
        if (step()) return true;
#pragma unroll 1
    for (uint32_t probe = kMaxProbe; probe < t.max_probe; probe++)
        if (step()) return true;
    return false;
}

__device__ __forceinline__ int ct_lookup(const CountTable &t, uint32_t key) {
    const uint32_t C = t.C;
    if (key == kEmptyKey) return t.cnt[C] ? (int)C : -1;
    uint32_t s = ct_home(key, C);
    for (uint32_t probe = 0; probe < kMaxProbe; probe++) {
        const uint32_t k = t.keys[s];
        if (k == key) return (int)s;
        if (k == kEmptyKey) return -1;
        s = s + 1 == C ? 0 : s + 1;
    }
#pragma unroll 1
    for (uint32_t probe = kMaxProbe; probe < t.max_probe; probe++) {
        const uint32_t k = t.keys[s];
        if (k == key) return (int)s;
        if (k == kEmptyKey) return -1;
        s = s + 1 == C ? 0 : s + 1;
    }
    return -1;
}

constexpr int kJoinPer = 8;   // elements per thread per tile (independent loads in flight)

// Probe tuples per join piece: at most kJoinChunk (a piece of a long run then
// ends within some 20 us of the others), at least kJoinChunkMin, or
// kJoinChunkEnum when pairs are enumerated.
constexpr uint32_t kJoinChunk = 65536;
constexpr uint32_t kJoinChunkMin = 2048, kJoinChunkEnum = 16384;
// Build and probe tuples of a raw-only call's items: at least kRawPiece; square
// pieces of up to kRawPieceMost, when they make one wave of CTAs.
constexpr uint32_t kRawPiece = 1024, kRawPieceMost = 4096;

// A run of tuples: (val << 32 | key) words of a partitioned array, or (kRaw)
// the key and val of 16-byte tuples.
template <bool kRaw>
__device__ __forceinline__ uint64_t run_load(const void *p, uint32_t i) {
    if (kRaw) {
        const uint2 v = __ldg(static_cast<const uint2 *>(p) + 2 * (size_t)i);
        return ((uint64_t)v.y << 32) | v.x;
    }
    return static_cast<const uint64_t *>(p)[i];
}

// Where an item's runs lie and which side builds.
struct JoinRuns {
    void *b;         // build run (a partitioned one may be compacted in place)
    const void *p;   // probe piece
    uint32_t bside;  // side of the build tuples: 0 left (fr), 1 right (gs); the probes have the other's hash
};
__device__ __forceinline__ JoinRuns join_runs(const JoinItem &ji, const sjbg_tuple *__restrict__ L,
                                              const sjbg_tuple *__restrict__ R, const WinPlan *__restrict__ wins,
                                              uint64_t *partL, uint64_t *partR) {
    JoinRuns r;
    const bool swap = (ji.flags & kItemSwap) != 0;
    r.bside = swap ? 1u : 0u;
    if (ji.flags & kItemRaw) {
        const sjbg_tuple *l = L + wins[ji.w].left_off, *t = R + wins[ji.w].right_off;
        r.b = const_cast<sjbg_tuple *>((swap ? t : l) + ji.sB);   // never written: every key of a raw window fits
        r.p = (swap ? l : t) + ji.sP;
    } else {
        r.b = (swap ? partR : partL) + ji.sB;
        r.p = (swap ? partL : partR) + ji.sP;
    }
    return r;
}

// The bucket's count table in shared memory (cap slots).
static inline size_t count_table_bytes(uint32_t cap) {
    return (sizeof(unsigned long long) + 2 * sizeof(uint32_t)) * ((size_t)cap + 1);
}

// ---- bucket join by places
// The build run is distributed over `places` short lists (about two tuples
// each) by a hash of the key: one pass counts the places, a scan gives their
// starts, a second pass writes the (key, val) words; a probe then compares the
// words of its key's place.  Two shared atomics per build tuple and two or
// three shared loads per probe, and nothing that grows with the table's load:
// the open-addressing table it replaced for these buckets (16-byte slots, a
// compare-and-swap and three atomics per build tuple, load up to 0.77) left a
// warp's lanes waiting for the longest walk, 9 of 32 active, even with a key
// filter in front.  A window of 65,536 tuples per side in 256 pieces of 4,096
// by 4,096: 82 us with the table, 24 us by places.
constexpr uint32_t kPlaceCap = 8192;      // build tuples
constexpr uint32_t kPlacesMax = 4096;
// Repeated keys leave the bucket to the hash table, which adds them up: by
// places a probe pays for every match, with a hash of the match's value.  The
// squares of the places' tuple numbers tell how many build tuples share a
// tuple's key on average: distinct keys give about nB + nB^2 / places, a key of
// k tuples k^2.  64 windows of 2^20, scattered keys, 1 / 2 / 3 / 4 / 8 tuples per
// key (a tuple then shares its key with 2 / 3 / 4 / 5 / 9): by places 1.91 / 2.09
// / 2.28 / 2.42 / 2.90 ms, by the table 2.39 / 2.08 / 1.97 / 1.90 / 1.80, so the
// line is at 3.5 (the try costs the table 1 to 4 %).  A few hot keys among
// distinct ones hold up their probes' warps before the mean shows them: a place
// of more than kPlaceMost decides too (z = 0.5: 64 windows of 2^20 without a
// limit 2.47, 32 2.38, 20 2.31, by the table alone 2.23; 1,024 of 30,000 1.54,
// 1.20, 1.13, 1.13; z = 0.25 64 of 2^20: 32 1.97, 20 1.98, 16 2.01, table 2.36).
constexpr uint32_t kPlaceRepeat2 = 7;   // twice the tuples that share a tuple's key
constexpr uint32_t kPlaceMost = 20;
constexpr size_t kPlaceBytes = sizeof(uint64_t) * kPlaceCap + sizeof(uint32_t) * (kPlacesMax + 1);

// Adds the matches to count and prod; false, with nothing added, when the run's
// keys repeat (nB <= kPlaceCap).  e: the build run's first tile (build_head).
template <bool kRaw>
__device__ __forceinline__ bool join_count_places(const JoinItem &ji, const JoinRuns &jr, uint64_t (&e)[kJoinPer],
                                                  unsigned long long &count, unsigned long long &prod) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ uint32_t warp_tot[kJoinThreads / 32], warp_sq[kJoinThreads / 32];
    uint64_t *word = reinterpret_cast<uint64_t *>(smem_raw);
    uint32_t *at = reinterpret_cast<uint32_t *>(word + kPlaceCap);   // at[p]: first word of place p; at[0] = 0
    const uint32_t nB = ji.nB, nP = ji.nP, bside = jr.bside, pside = bside ^ 1u;
    const uint32_t bits = min(12u, max(9u, 31u - (uint32_t)__clz(nB))), places = 1u << bits, shift = 32u - bits;
    static_assert(kPlacesMax == 1u << 12 && kJoinThreads == 1 << 9, "places per thread");
    auto load = [&](uint32_t base) {
#pragma unroll
        for (int k = 0; k < kJoinPer; k++) {
            const uint32_t i = base + k * kJoinThreads + threadIdx.x;
            e[k] = i < nB ? run_load<kRaw>(jr.b, i) : 0ull;
        }
    };
    constexpr uint32_t tile = kJoinPer * kJoinThreads;
    for (uint32_t i = threadIdx.x; i <= places; i += kJoinThreads) at[i] = 0;
    SJBG_BARRIER();
    for (uint32_t base = 0; base < nB; base += tile) {
        if (base) load(base);
#pragma unroll
        for (int k = 0; k < kJoinPer; k++)
            if (base + k * kJoinThreads + threadIdx.x < nB) atomicAdd(&at[1 + (place_hash((uint32_t)e[k]) >> shift)], 1u);
    }
    SJBG_BARRIER();
    const uint32_t per = places / kJoinThreads, p0 = 1 + threadIdx.x * per;   // 1 to 8 places
    uint32_t sum = 0, squares = 0, largest = 0;   // (squares of at most kPlaceCap tuples: 2^26)
    for (uint32_t q = 0; q < per; q++) {
        const uint32_t c = at[p0 + q];
        sum += c;
        squares += c * c;
        largest = max(largest, c);
    }
    uint32_t tot;
    uint32_t run = warp_excl_scan(sum, &tot);
    squares = __reduce_add_sync(0xFFFFFFFFu, squares);
    if (lane_id() == 31) {
        warp_tot[warp_id()] = tot;
        warp_sq[warp_id()] = squares;
    }
    const bool most = __syncthreads_or(largest > kPlaceMost);
    squares = __reduce_add_sync(0xFFFFFFFFu, lane_id() < kJoinThreads / 32 ? warp_sq[lane_id()] : 0u);
    if (most || 2 * (squares - (nB * nB >> bits)) > kPlaceRepeat2 * nB) {   // (the same for the whole CTA)
        SJBG_BARRIER();   // the places are read before the next table's entries
        return false;
    }
    run += __reduce_add_sync(0xFFFFFFFFu, lane_id() < warp_id() ? warp_tot[lane_id() & (kJoinThreads / 32 - 1)] : 0u);
    for (uint32_t q = 0; q < per; q++) {
        const uint32_t c = at[p0 + q];
        at[p0 + q] = run;   // the place's next free word, in the end the next place's first
        run += c;
    }
    SJBG_BARRIER();
    for (uint32_t base = 0; base < nB; base += tile) {
        if (nB > tile) load(base);
#pragma unroll
        for (int k = 0; k < kJoinPer; k++)
            if (base + k * kJoinThreads + threadIdx.x < nB)
                word[atomicAdd(&at[1 + (place_hash((uint32_t)e[k]) >> shift)], 1u)] = e[k];
    }
    constexpr int kProbe = 4;
    uint64_t ahead[kProbe];
    auto probes = [&](uint32_t base) {
#pragma unroll
        for (int k = 0; k < kProbe; k++) {
            const uint32_t i = base + k * kJoinThreads + threadIdx.x;
            ahead[k] = i < nP ? run_load<kRaw>(jr.p, i) : 0ull;
        }
    };
    probes(0);
    SJBG_BARRIER();
    // kProbe probes of a thread at a time, step by step for all of them: the
    // bounds of their places, the first two words of each, and what is left of
    // longer ones.  The hash of a matching word is taken after the compares, once
    // per probe instead of once per compare that matches in some lane.  (1,024
    // windows of 2^10 to 2^20: 1,681 -> 1,470 us, one probe at a time before;
    // with the hash table out of line as well, 1,406; with the
    // next four loaded a step ahead, the first during the build, 1,283.)
    for (uint32_t base = 0; base < nP; base += kProbe * kJoinThreads) {
        uint64_t pr[kProbe], x0[kProbe], x1[kProbe];
        uint32_t j[kProbe], end[kProbe];
#pragma unroll
        for (int k = 0; k < kProbe; k++) pr[k] = ahead[k];
        probes(base + kProbe * kJoinThreads);
#pragma unroll
        for (int k = 0; k < kProbe; k++) {
            const uint32_t q = place_hash((uint32_t)pr[k]) >> shift;
            j[k] = at[q];
            end[k] = base + k * kJoinThreads + threadIdx.x < nP ? at[q + 1] : 0u;
        }
#pragma unroll
        for (int k = 0; k < kProbe; k++) {
            x0[k] = j[k] < end[k] ? word[j[k]] : 0ull;
            x1[k] = j[k] + 1 < end[k] ? word[j[k] + 1] : 0ull;
        }
#pragma unroll
        for (int k = 0; k < kProbe; k++) {
            const uint32_t key = (uint32_t)pr[k];
            uint32_t c = 0, m = 0;
            unsigned long long f = 0;
            auto compare = [&](uint64_t x, bool in) {
                if (in && (uint32_t)x == key) {
                    if (c++) f += sjbg_fside((uint32_t)(x >> 32), bside);
                    else m = (uint32_t)(x >> 32);
                }
            };
            compare(x0[k], j[k] < end[k]);
            compare(x1[k], j[k] + 1 < end[k]);
            for (uint32_t i = j[k] + 2; i < end[k]; i++) compare(word[i], true);
            if (c) {
                count += c;
                prod += (f + sjbg_fside(m, bside)) * sjbg_fside((uint32_t)(pr[k] >> 32), pside);
            }
        }
    }
    SJBG_BARRIER();   // the words are read before the next item's
    return true;
}

// Larger buckets (a radix window's hot keys) keep the hash table when they need
// a second direct pass, which re-reads the bucket; every build run of more than
// kPlaceCap tuples does, and its range is not looked for.
constexpr uint32_t kDirectMaxRun = 16384;

struct KeyRange {
    uint32_t lo, hi;
};

// The smallest lo and the largest hi of the CTA's threads, to every thread; its
// only barrier ends it after the CTA's first call (turn 0): the calls take the
// two result slots in turn and leave the other one reset.  (Not a template: raw
// and partitioned items of a CTA use the same slots.)
__device__ __forceinline__ KeyRange cta_key_range(uint32_t lo, uint32_t hi, uint32_t &turn) {
    __shared__ uint32_t min_s[2], max_s[2];
    if (turn == 0) {
        if (threadIdx.x == 0) {
            min_s[0] = min_s[1] = 0xFFFFFFFFu;
            max_s[0] = max_s[1] = 0;
        }
        SJBG_BARRIER();
    }
    const uint32_t slot = turn & 1u;
    turn = slot + 1;
    lo = __reduce_min_sync(0xFFFFFFFFu, lo);
    hi = __reduce_max_sync(0xFFFFFFFFu, hi);
    if (lane_id() == 0) {
        atomicMin(&min_s[slot], lo);
        atomicMax(&max_s[slot], hi);
    }
    SJBG_BARRIER();
    if (threadIdx.x == 0) {
        min_s[slot ^ 1u] = 0xFFFFFFFFu;
        max_s[slot ^ 1u] = 0;
    }
    return KeyRange{min_s[slot], max_s[slot]};
}

// Loads the first tile of a build run (kJoinPer tuples per thread) and returns
// the run's smallest and largest keys to every thread.
template <bool kRaw>
__device__ __forceinline__ KeyRange build_head(const JoinItem &ji, const JoinRuns &jr, uint64_t (&e)[kJoinPer],
                                               uint32_t &turn) {
    uint32_t lo = 0xFFFFFFFFu, hi = 0;
#pragma unroll
    for (int k = 0; k < kJoinPer; k++) {
        const uint32_t i = k * kJoinThreads + threadIdx.x;
        e[k] = i < ji.nB ? run_load<kRaw>(jr.b, i) : 0ull;
    }
#pragma unroll
    for (int k = 0; k < kJoinPer; k++) {
        if (k * kJoinThreads + threadIdx.x < ji.nB) {
            lo = min(lo, (uint32_t)e[k]);
            hi = max(hi, (uint32_t)e[k]);
        }
    }
    for (uint32_t i = kJoinPer * kJoinThreads + threadIdx.x; i < ji.nB; i += kJoinThreads) {
        const uint32_t key = (uint32_t)run_load<kRaw>(jr.b, i);
        lo = min(lo, key);
        hi = max(hi, key);
    }
    return cta_key_range(lo, hi, turn);
}

template <bool kRaw>
__device__ __forceinline__ void join_count_bucket(const JoinItem &ji, const JoinRuns &jr, uint32_t cap,
                                                  unsigned long long &count, unsigned long long &prod) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ uint32_t novf;
    const uint32_t nB = ji.nB, nP = ji.nP;
    const uint32_t bside = jr.bside, pside = bside ^ 1u;
    // the table holds at most nB distinct keys: 2 slots per build tuple (at
    // least 64, at most the launch's capacity of 1.3 per target tuple, which
    // lets two CTAs share an SM), so buckets under the target probe at load
    // <= 1/2: with mostly distinct keys a miss then walks ~3 slots, not ~10
    const uint32_t C = min(cap, max(64u, (nB * 2u + 31u) & ~31u));
    CountTable t;
    t.sumf = reinterpret_cast<unsigned long long *>(smem_raw);
    t.keys = reinterpret_cast<uint32_t *>(t.sumf + C + 1);
    t.cnt = t.keys + C + 1;
    t.C = C;
    t.max_probe = nB < C ? C : kMaxProbe;
    constexpr uint32_t tile = kJoinPer * kJoinThreads;

    uint64_t e[kJoinPer];
    uint32_t n = nB;
    for (;;) {
        for (uint32_t i = threadIdx.x; i <= C; i += kJoinThreads) {
            t.keys[i] = kEmptyKey;
            t.cnt[i] = 0;
            t.sumf[i] = 0;
        }
        if (threadIdx.x == 0) novf = 0;
        SJBG_BARRIER();
        // build: kJoinPer independent loads per thread, then insert them
        for (uint32_t base = 0; base < n; base += tile) {
#pragma unroll
            for (int k = 0; k < kJoinPer; k++) {
                const uint32_t i = base + k * kJoinThreads + threadIdx.x;
                e[k] = i < n ? run_load<kRaw>(jr.b, i) : 0ull;
            }
            SJBG_BARRIER();   // every read of this tile precedes any overflow write
#pragma unroll
            for (int k = 0; k < kJoinPer; k++) {
                const uint32_t i = base + k * kJoinThreads + threadIdx.x;
                const bool valid = i < n;
                const bool ok = !valid || ct_insert(t, (uint32_t)e[k], 1u, sjbg_fside((uint32_t)(e[k] >> 32), bside));
                // (a piece's table, and a raw window's, takes every key: nothing is written back)
                if (!kRaw && valid && !ok) static_cast<uint64_t *>(jr.b)[atomicAdd(&novf, 1u)] = e[k];
                __syncwarp();
            }
        }
        SJBG_BARRIER();
        // probe: the same independent-load tiling, no barriers needed
        for (uint32_t base = 0; base < nP; base += tile) {
#pragma unroll
            for (int k = 0; k < kJoinPer; k++) {
                const uint32_t j = base + k * kJoinThreads + threadIdx.x;
                e[k] = j < nP ? run_load<kRaw>(jr.p, j) : ~0ull;
            }
#pragma unroll
            for (int k = 0; k < kJoinPer; k++) {
                const uint32_t j = base + k * kJoinThreads + threadIdx.x;
                if (j < nP) {
                    const int s = ct_lookup(t, (uint32_t)e[k]);
                    if (s >= 0) {
                        count += t.cnt[s];
                        prod += t.sumf[s] * sjbg_fside((uint32_t)(e[k] >> 32), pside);
                    }
                }
                __syncwarp();
            }
        }
        SJBG_BARRIER();
        n = novf;
        SJBG_BARRIER();
        if (n == 0) break;
    }
}

// A pair of pieces of a bucket whose build run is longer than its table (a hot
// key's tuples, or those of many keys).  Other CTAs read the same runs, so
// nothing is compacted: when a key finds no slot, the pieces are joined again
// in twice as many passes, each over the keys of one residue of a mixed key,
// until every pass fits.  A warp adds the tuples of its first lane's key at
// once when they are many: same-address shared atomics take the lanes in turn.
__device__ __noinline__ void join_count_hot(const uint64_t *b, uint32_t nB, const uint64_t *p, uint32_t nP,
                                            uint32_t bside, WinAcc *acc, uint32_t C) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ uint32_t refused;
    CountTable t;
    t.sumf = reinterpret_cast<unsigned long long *>(smem_raw);
    t.keys = reinterpret_cast<uint32_t *>(t.sumf + C + 1);
    t.cnt = t.keys + C + 1;
    t.C = C;
    t.max_probe = kMaxProbe;
    auto residue = [](uint32_t key, uint32_t passes) {   // of a bijection of the key
        uint32_t x = key * 0x85EBCA6Bu;
        x ^= x >> 16;
        return x & (passes - 1);
    };
    unsigned long long count = 0, prod = 0;
    bool done = false;
    for (uint32_t passes = 1; !done && passes < (1u << 31); passes <<= 1) {
        count = prod = 0;
        done = true;
        for (uint32_t s = 0; s < passes && done; s++) {
            for (uint32_t i = threadIdx.x; i <= C; i += kJoinThreads) {
                t.keys[i] = kEmptyKey;
                t.cnt[i] = 0;
                t.sumf[i] = 0;
            }
            if (threadIdx.x == 0) refused = 0;
            SJBG_BARRIER();
            for (uint32_t base = 0; base < nB; base += 4 * kJoinThreads) {
                uint64_t e[4];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const uint32_t i = base + k * kJoinThreads + threadIdx.x;
                    e[k] = i < nB ? b[i] : 0ull;
                }
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const uint32_t key = (uint32_t)e[k];
                    bool in = base + k * kJoinThreads + threadIdx.x < nB && residue(key, passes) == s;
                    unsigned long long f = sjbg_fside((uint32_t)(e[k] >> 32), bside);
                    uint32_t c = 1;
                    const uint32_t key0 = __shfl_sync(0xFFFFFFFFu, key, 0);   // (every lane: not inside the &&)
                    const bool same = in && key == key0;
                    const unsigned grp = __ballot_sync(0xFFFFFFFFu, same);
                    if (__popc(grp) >= 8) {   // the first lane's group as one
                        const unsigned long long sum = warp_sum_u64(same ? f : 0ull);
                        if (same) {
                            in = (int)lane_id() == __ffs(grp) - 1;
                            f = sum;
                            c = __popc(grp);
                        }
                    }
                    if (in && !ct_insert(t, key, c, f)) refused = 1;
                }
            }
            SJBG_BARRIER();
            done = refused == 0;
            if (done) {
                for (uint32_t base = 0; base < nP; base += 4 * kJoinThreads) {
                    uint64_t e[4];
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const uint32_t i = base + k * kJoinThreads + threadIdx.x;
                        e[k] = i < nP ? p[i] : 0ull;
                    }
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const uint32_t key = (uint32_t)e[k];
                        if (base + k * kJoinThreads + threadIdx.x >= nP || residue(key, passes) != s) continue;
                        const int x = ct_lookup(t, key);
                        if (x >= 0) {
                            count += t.cnt[x];
                            prod += t.sumf[x] * sjbg_fside((uint32_t)(e[k] >> 32), bside ^ 1u);
                        }
                    }
                }
            }
            SJBG_BARRIER();   // the table and `refused` are read before they are reset
        }
    }
    flush_acc(acc, count, 0, prod);
}

// ---- direct-addressed bucket join
// In a radix window every key of bucket b has key & (2^lg - 1) == b, so key >> lg
// tells the bucket's keys apart (lg = 0 in a window that is not partitioned).
// When the build run's indices key >> lg span few values the build side is a
// direct table {count, hash sum} indexed from the smallest one: an insert is
// three shared atomics and a probe two loads, with no key compares or probe
// loop (the hash table spends about 120 thread instructions per tuple there,
// and is issue- and shared-memory-bound).  A pass covers kDirectMax indices; a
// bucket whose indices need more than kDirectPasses passes goes through the
// hash table: the build run's smallest and largest keys, found while its first
// tile is loaded, decide.  (Learned buckets, which are key ranges, gained
// nothing: their probes match, and the range costs a barrier to find.)
// Measured on 1,024 uneven windows (keys in [0, 4W), about 4,096 left tuples
// per bucket, two passes): the bucket joins take 2.02 ms, against 2.91 ms with
// hash tables.
constexpr uint32_t kDirectMax = 8192;
constexpr uint32_t kDirectPasses = 2;
// A build run of at most kDirectSave tuples keeps each tuple's table index (16
// bits, 0xFFFF outside the pass's range) in shared memory during the build, so
// the table is reset from there instead of from a second read of the run.
constexpr uint32_t kDirectSave = 4096;
constexpr size_t kDirectBytes =
    (sizeof(unsigned long long) + sizeof(uint32_t)) * kDirectMax + sizeof(uint16_t) * kDirectSave;

// Passes of a bucket whose build run has keys in kr, or 0: the hash table.
__device__ __forceinline__ uint32_t direct_passes(const JoinItem &ji, KeyRange kr) {
    const uint32_t passes = ((kr.hi >> ji.lg) - (kr.lo >> ji.lg)) / kDirectMax + 1;
    if (passes > kDirectPasses || (passes > 1 && ji.nB + ji.nP > kDirectMaxRun)) return 0;
    return passes;
}

// `clean`: the leading table entries known to be zero (CTA-uniform); a direct
// bucket leaves the table zero again, a hash-table bucket does not.  e: the
// build run's first tile (build_head); first: its smallest index.  The matches
// are added to count and prod, as in join_count_bucket.
template <bool kRaw>
__device__ __forceinline__ void join_count_direct(const JoinItem &ji, const JoinRuns &jr, uint64_t (&e)[kJoinPer],
                                                  uint32_t first, uint32_t passes, uint32_t &clean,
                                                  unsigned long long &count, unsigned long long &prod) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    const uint32_t nB = ji.nB, nP = ji.nP, lg = ji.lg;
    const uint32_t bside = jr.bside, pside = bside ^ 1u;
    unsigned long long *dsum = reinterpret_cast<unsigned long long *>(smem_raw);
    uint32_t *dcnt = reinterpret_cast<uint32_t *>(dsum + kDirectMax);
    uint16_t *dsave = reinterpret_cast<uint16_t *>(dcnt + kDirectMax);   // kDirectSave indices
    const bool save = nB <= kDirectSave;
    for (uint32_t i = clean + threadIdx.x; i < kDirectMax; i += kJoinThreads) {
        dsum[i] = 0;
        dcnt[i] = 0;
    }
    if (clean != kDirectMax) SJBG_BARRIER();
    clean = kDirectMax;
    constexpr uint32_t tile = kJoinPer * kJoinThreads;
    for (uint32_t p = 0; p < passes; p++) {
        const uint32_t lo = first + p * kDirectMax;
        // build: the build keys whose index falls in [lo, lo + kDirectMax)
        for (uint32_t base = 0; base < nB; base += tile) {
            if (p || base) {
#pragma unroll
                for (int k = 0; k < kJoinPer; k++) {
                    const uint32_t i = base + k * kJoinThreads + threadIdx.x;
                    e[k] = i < nB ? run_load<kRaw>(jr.b, i) : 0ull;
                }
            }
#pragma unroll
            for (int k = 0; k < kJoinPer; k++) {
                const uint32_t i = base + k * kJoinThreads + threadIdx.x;
                if (i < nB) {
                    const uint32_t d = ((uint32_t)e[k] >> lg) - lo;   // wraps for indices below the range
                    if (save) dsave[i] = d < kDirectMax ? (uint16_t)d : (uint16_t)0xFFFFu;
                    if (d < kDirectMax) {
                        atomicAdd(&dcnt[d], 1u);
                        ct_add_sum(&dsum[d], sjbg_fside((uint32_t)(e[k] >> 32), bside));
                    }
                }
            }
        }
        SJBG_BARRIER();
        // probe: the probe keys in the range
        for (uint32_t base = 0; base < nP; base += tile) {
            uint64_t q[kJoinPer];
#pragma unroll
            for (int k = 0; k < kJoinPer; k++) {
                const uint32_t j = base + k * kJoinThreads + threadIdx.x;
                q[k] = j < nP ? run_load<kRaw>(jr.p, j) : 0ull;
            }
#pragma unroll
            for (int k = 0; k < kJoinPer; k++) {
                const uint32_t d = ((uint32_t)q[k] >> lg) - lo;
                if (base + k * kJoinThreads + threadIdx.x < nP && d < kDirectMax) {
                    const uint32_t c = dcnt[d];
                    if (c) {
                        count += c;
                        prod += dsum[d] * sjbg_fside((uint32_t)(q[k] >> 32), pside);
                    }
                }
            }
        }
        SJBG_BARRIER();
        // leave the table zero: the range's build entries (their saved indices,
        // or for a longer run the run again, from L2)
        for (uint32_t i = threadIdx.x; i < nB; i += kJoinThreads) {
            const uint32_t d = save ? (uint32_t)dsave[i] : ((uint32_t)run_load<kRaw>(jr.b, i) >> lg) - lo;
            if (d < kDirectMax) {
                dcnt[d] = 0;
                dsum[d] = 0;
            }
        }
        SJBG_BARRIER();
    }
}

constexpr uint32_t kEnumChunk = 4096;  // left tuples per chained chunk
constexpr uint32_t kNil = 0xFFFFFFFFu;

__device__ __forceinline__ void join_enum_bucket(const JoinItem &ji, const uint64_t *__restrict__ partL,
                                                 const uint64_t *__restrict__ partR, WinAcc *__restrict__ acc,
                                                 const WinPlan *__restrict__ wins, sjbg_pair *__restrict__ pairs,
                                                 uint32_t table_bits) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    const uint32_t nR = ji.nB, nS = ji.nP;   // (enumerating joins build from the left)
    if (nR == 0 || nS == 0) return;
    const uint64_t *Rb = partL + ji.sB;
    const uint64_t *Sb = partR + ji.sP;
    const uint32_t w = ji.w;
    const uint32_t Cmax = 1u << table_bits;
    uint32_t *keys = reinterpret_cast<uint32_t *>(smem_raw);   // Cmax + 1
    uint32_t *head = keys + Cmax + 1;                          // Cmax + 1
    uint32_t *next = head + Cmax + 1;                          // kEnumChunk
    uint32_t *vals = next + kEnumChunk;                        // kEnumChunk
    const uint64_t pcap = pairs ? wins[w].pairs_cap : 0;
    sjbg_pair *pout = pairs ? pairs + wins[w].pairs_off : nullptr;

    unsigned long long count = 0, prod = 0, xr = 0;
    for (uint32_t c0 = 0; c0 < nR; c0 += kEnumChunk) {
        const uint32_t m = min(kEnumChunk, nR - c0);
        // at least twice as many slots as the chunk has tuples (slot C holds key 0xFFFFFFFF)
        uint32_t bits = 6;
        while (bits < table_bits && (1u << bits) < 2 * m) bits++;
        const uint32_t C = 1u << bits;
        for (uint32_t i = threadIdx.x; i <= C; i += blockDim.x) {
            keys[i] = kEmptyKey;
            head[i] = kNil;
        }
        SJBG_BARRIER();
        // insert: the trip count is uniform per block (bounds checked inside), and
        // every warp reconverges before the barrier
        for (uint32_t i0 = 0; i0 < m; i0 += blockDim.x) {
            const uint32_t i = i0 + threadIdx.x;
            if (i < m) {
                const uint64_t e = Rb[c0 + i];
                const uint32_t key = (uint32_t)e;
                vals[i] = (uint32_t)(e >> 32);
                uint32_t s;
                if (key == kEmptyKey) {
                    s = C;
                } else {
                    s = slot_hash(key, bits);
                    // at most m <= C/2 keys: a free or matching slot exists within C probes
                    for (uint32_t p = 0; p < C; p++) {
                        const uint32_t prev = atomicCAS(&keys[s], kEmptyKey, key);
                        if (prev == kEmptyKey || prev == key) break;
                        s = (s + 1) & (C - 1);
                    }
                }
                next[i] = atomicExch(&head[s], i);
            }
            __syncwarp();
        }
        SJBG_BARRIER();
        // probe: loop bound is uniform per warp so the pair reservation can use shuffles
        for (uint32_t j0 = 0; j0 < nS; j0 += blockDim.x) {
            const uint32_t j = j0 + threadIdx.x;
            uint32_t h = kNil, sv = 0;
            if (j < nS) {
                const uint64_t e = Sb[j];
                const uint32_t key = (uint32_t)e;
                sv = (uint32_t)(e >> 32);
                uint32_t s = kNil;
                if (key == kEmptyKey) {
                    s = C;
                } else {
                    uint32_t q = slot_hash(key, bits);
                    for (uint32_t p = 0; p <= C; p++) {
                        const uint32_t k = keys[q];
                        if (k == key) { s = q; break; }
                        if (k == kEmptyKey) break;
                        q = (q + 1) & (C - 1);
                    }
                }
                if (s != kNil) h = head[s];
            }
            uint32_t mine = 0;
            const unsigned long long gs = sjbg_gs(sv);
            // chains link indices of this chunk: a walk never takes more than m steps
            for (uint32_t i = h, steps = 0; i < m && steps < m; i = next[i], steps++) {
                const uint32_t rv = vals[i];
                xr ^= sjbg_pair_hash(rv, sv);
                prod += sjbg_fr(rv) * gs;
                mine++;
            }
            count += mine;
            if (pout) {
                uint32_t tot;
                const uint32_t ex = warp_excl_scan(mine, &tot);
                unsigned long long base = 0;
                if (lane_id() == 0 && tot) base = atomicAdd(&acc[w].npairs, (unsigned long long)tot);
                base = __shfl_sync(0xFFFFFFFFu, base, 0) + ex;
                for (uint32_t i = h, steps = 0; i < m && steps < m; i = next[i], steps++) {
                    if (base < pcap) pout[base] = sjbg_pair{vals[i], sv};
                    base++;
                }
            }
            __syncwarp();
        }
        SJBG_BARRIER();
    }
    flush_acc(&acc[w], count, xr, prod);
}

// The hash table for what neither a direct table nor the places take: out of
// line, so that the code of the usual items stays short (and by value, so that
// nothing of theirs lives in local memory).
struct JoinSums {
    unsigned long long count, prod;
};
template <bool kRaw>
__device__ __noinline__ JoinSums join_count_rest(const JoinItem ji, const JoinRuns jr, uint32_t cap) {
    JoinSums r{0, 0};
    join_count_bucket<kRaw>(ji, jr, cap, r.count, r.prod);
    return r;
}

// One item's matches; `clean` as in join_count_direct, `turn` as in build_head
// (0 at the CTA's first item).
template <bool kRaw, bool kModels>
__device__ __forceinline__ void join_item(const JoinItem &ji, const JoinRuns &jr, uint32_t cap, uint32_t &clean,
                                          uint32_t &turn, unsigned long long &count, unsigned long long &prod) {
    // a learned bucket's light keys are a range (no direct table) and repeat, up
    // to the heavy cut: the hash table, which aggregates them (z = 1.5, 8 x 2^24:
    // 54 us, by places 130)
    if (kModels && (ji.flags & kItemModel)) {
        join_count_bucket<kRaw>(ji, jr, cap, count, prod);
        clean = 0;
        return;
    }
    uint64_t e[kJoinPer];
    if (ji.nB <= kPlaceCap) {
        const KeyRange kr = build_head<kRaw>(ji, jr, e, turn);
        if (const uint32_t passes = direct_passes(ji, kr)) {
            join_count_direct<kRaw>(ji, jr, e, kr.lo >> ji.lg, passes, clean, count, prod);
            return;
        }
    }
    clean = 0;
    if (ji.nB <= kPlaceCap && join_count_places<kRaw>(ji, jr, e, count, prod)) return;
    const JoinSums r = join_count_rest<kRaw>(ji, jr, cap);
    count += r.count;
    prod += r.prod;
}

// ---- joins from sorted tiles
// Buckets of windows joined from sorted tiles: a bucket is the runs of all
// tiles of the window, the left side's tiles first.  Their words are numbered
// across the runs (owner: the tile of each of kRowsOwner words at a time), so
// that every lane has one; the smaller side's words build a count table, the
// others probe it.  Words whose keys the table cannot take are written back over
// the first words of their side (this CTA's alone) and joined in a further pass.  Part of the
// bucket join's launch: persistent CTAs over work kind 4.
constexpr uint32_t kRowsOwner = 4096;
constexpr uint32_t kRowsRun = 64;   // a longer run: the owners are written by warps, not by threads
struct RowsLists {
    uint32_t pre[kRowsTilesMax + 1];    // words of the bucket in the tiles before
    uint16_t off[kRowsTilesMax];        // its run in the tile
    uint16_t owner[kRowsOwner];
};
static inline size_t rows_join_bytes(uint32_t cap) { return ((count_table_bytes(cap) + 15) & ~(size_t)15) + sizeof(RowsLists); }

struct RowsJoin {
    uint32_t nwin, rstride;
    const uint32_t *tileL, *tileR, *work, *ccnt;
    uint64_t *compL, *compR;
    const uint16_t *rows16;
    uint32_t *queue;   // null: no window of the call may take the form
};

__device__ __forceinline__ void rows_join(const RowsJoin &rj, const WinPlan *__restrict__ wins, WinAcc *__restrict__ acc,
                                          uint32_t cap) {
    const uint32_t nwin = rj.nwin, rstride = rj.rstride;
    const uint32_t *__restrict__ tileL = rj.tileL, *__restrict__ tileR = rj.tileR, *__restrict__ ccnt = rj.ccnt;
    uint64_t *compL = rj.compL, *compR = rj.compR;
    const uint16_t *__restrict__ rows16 = rj.rows16;
    uint32_t *queue = rj.queue;
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ uint32_t warp_tot[32];
    __shared__ uint32_t next_s, novf_s, n_left_s;
    RowsLists &ls = *reinterpret_cast<RowsLists *>(smem_raw + ((sizeof(unsigned long long) + 2 * sizeof(uint32_t)) *
                                                                   ((size_t)cap + 1) + 15 & ~(size_t)15));
    const uint32_t *pw = rj.work + 2 * kWorkRows * (nwin + 1);
    const uint32_t items = pw[nwin];
    uint32_t g = blockIdx.x;
    while (g < items) {
        uint32_t claim = 0;
        if (threadIdx.x == 0) claim = gridDim.x + atomicAdd(queue, 1u);
        const uint32_t w = find_window(pw, nwin, g), b = g - pw[w];
        const uint32_t TL = (ccnt[2 * w] + kTile - 1) / kTile, T = TL + (ccnt[2 * w + 1] + kTile - 1) / kTile;
        uint64_t *wl = compL + (uint64_t)tileL[w] * kTile, *wr = compR + (uint64_t)tileR[w] * kTile;
        const uint16_t *rl = rows16 + (uint64_t)tileL[w] * rstride + b;
        const uint16_t *rr = rows16 + ((uint64_t)tileL[nwin] + tileR[w]) * rstride + b;
        // thread t's tiles [t * per, t * per + per)
        constexpr uint32_t kPerMax = kRowsTilesMax / kJoinThreads;
        const uint32_t per = (T + kJoinThreads - 1) / kJoinThreads, x0 = threadIdx.x * per;
        uint32_t sum = 0;
        bool lengthy = false;
        uint32_t len[kPerMax];
#pragma unroll
        for (uint32_t q = 0; q < kPerMax; q++) {
            const uint32_t x = x0 + q;
            len[q] = 0;
            if (q < per && x < T) {
                const uint16_t *r = x < TL ? rl + (uint64_t)x * rstride : rr + (uint64_t)(x - TL) * rstride;
                const uint32_t o = __ldg(r);
                len[q] = __ldg(r + 1) - o;
                ls.off[x] = (uint16_t)o;
            }
            sum += len[q];
            lengthy |= len[q] > kRowsRun;
        }
        lengthy = __any_sync(0xFFFFFFFFu, lengthy);
        uint32_t tot;
        uint32_t run = warp_excl_scan(sum, &tot);
        if (lane_id() == 31) warp_tot[warp_id()] = tot | (lengthy ? 1u << 31 : 0u);   // (at most kRowsTilesMax * kTile)
        SJBG_BARRIER();
        uint32_t v = lane_id() < kJoinThreads / 32 ? warp_tot[lane_id()] : 0u;
        lengthy = __any_sync(0xFFFFFFFFu, v >> 31);
        v &= 0x7FFFFFFFu;
        const uint32_t n = __reduce_add_sync(0xFFFFFFFFu, v);
        run += __reduce_add_sync(0xFFFFFFFFu, lane_id() < warp_id() ? v : 0u);
#pragma unroll
        for (uint32_t q = 0; q < kPerMax; q++) {
            const uint32_t x = x0 + q;
            if (q < per && x < T) {
                ls.pre[x] = run;
                if (x == TL) n_left_s = run;
            }
            run += len[q];
        }
        if (TL == T && threadIdx.x == 0) n_left_s = n;
        if (threadIdx.x == 0) ls.pre[T] = n;
        SJBG_BARRIER();
        const uint32_t nl = n_left_s;
        auto tile_of = [&](uint32_t x) { return x < TL ? wl + (uint64_t)x * kTile : wr + (uint64_t)(x - TL) * kTile; };
        // words [i0, i1) of the bucket, kRowsOwner at a time; use(word) by every lane
        // that has one (build: once all lanes have loaded theirs)
        auto each = [&](uint32_t i0, uint32_t i1, auto build, auto use) {
            for (uint32_t c0 = i0; c0 < i1; c0 += kRowsOwner) {
                const uint32_t c1 = min(i1, c0 + kRowsOwner);
                if (lengthy) {   // a warp per run
                    for (uint32_t x = warp_id(); x < T; x += kJoinThreads / 32) {
                        const uint32_t a = max(ls.pre[x], c0), z = min(ls.pre[x + 1], c1);
                        for (uint32_t i = a + lane_id(); i < z; i += 32) ls.owner[i - c0] = (uint16_t)x;
                    }
                } else {         // a thread per run
                    for (uint32_t q = 0; q < per; q++) {
                        const uint32_t x = x0 + q;
                        if (x >= T) break;
                        const uint32_t a = max(ls.pre[x], c0), z = min(ls.pre[x + 1], c1);
                        for (uint32_t i = a; i < z; i++) ls.owner[i - c0] = (uint16_t)x;
                    }
                }
                SJBG_BARRIER();
                // (the trip count is uniform per CTA, and every warp reconverges after each use)
                for (uint32_t i0 = c0; i0 < c1; i0 += 4 * kJoinThreads) {
                    const uint32_t i = i0 + threadIdx.x;
                    uint64_t e[4];
#pragma unroll
                    for (uint32_t q = 0; q < 4; q++) {
                        const uint32_t k = i + q * kJoinThreads;
                        e[q] = 0;
                        if (k < c1) {
                            const uint32_t x = ls.owner[k - c0], at = ls.off[x] + (k - ls.pre[x]);
                            e[q] = build() ? tile_of(x)[at] : __ldg(tile_of(x) + at);
                        }
                    }
                    if constexpr (build()) SJBG_BARRIER();
#pragma unroll
                    for (uint32_t q = 0; q < 4; q++) {
                        if (i + q * kJoinThreads < c1) use(e[q]);
                        __syncwarp();
                    }
                }
                SJBG_BARRIER();   // (the owners are read before the next ones are written)
            }
        };
        if (nl != 0 && nl != n) {   // (the same for the whole CTA)
            CountTable t;
            const uint32_t right = n - nl < nl, nb = right ? n - nl : nl;   // built from the smaller side
            const uint32_t b0 = right ? nl : 0u, p0 = nl - b0, p1 = right ? nl : n;
            t.C = min(cap, max(64u, (nb * 2u + 31u) & ~31u));
            t.max_probe = kMaxProbe;   // (crowded homes are cheaper to join in a further pass)
            t.sumf = reinterpret_cast<unsigned long long *>(smem_raw);
            t.keys = reinterpret_cast<uint32_t *>(t.sumf + t.C + 1);
            t.cnt = t.keys + t.C + 1;
            unsigned long long count = 0, prod = 0;
            for (uint32_t rem = nb; rem;) {
                for (uint32_t i = threadIdx.x; i <= t.C; i += kJoinThreads) {
                    t.keys[i] = kEmptyKey;
                    t.cnt[i] = 0;
                    t.sumf[i] = 0;
                }
                if (threadIdx.x == 0) novf_s = 0;
                SJBG_BARRIER();
                each(b0, b0 + rem, std::true_type{}, [&](uint64_t e) {
                    if (ct_insert(t, (uint32_t)e, 1u, sjbg_fside((uint32_t)(e >> 32), right))) return;
                    const uint32_t k = b0 + atomicAdd(&novf_s, 1u);   // (no further than the words read so far)
                    uint32_t x0 = right ? TL : 0u, x1 = right ? T : TL;   // the last tile with its first word at or before k
                    while (x1 - x0 > 1) {
                        const uint32_t xm = (x0 + x1) / 2;
                        if (ls.pre[xm] <= k) x0 = xm;
                        else x1 = xm;
                    }
                    tile_of(x0)[ls.off[x0] + (k - ls.pre[x0])] = e;
                });   // ends with a barrier
                each(p0, p1, std::false_type{}, [&](uint64_t e) {
                    const int s = ct_lookup(t, (uint32_t)e);
                    if (s >= 0) {
                        count += t.cnt[s];
                        prod += t.sumf[s] * sjbg_fside((uint32_t)(e >> 32), right ^ 1u);
                    }
                });   // ends with a barrier
                rem = novf_s;
                SJBG_BARRIER();   // read before it is reset
            }
            flush_acc(&acc[w], count, 0, prod);
        }
        if (threadIdx.x == 0) next_s = claim;
        SJBG_BARRIER();
        g = next_s;
        SJBG_BARRIER();   // read before the next claim is stored
    }
}

// Bucket joins over the join list (items, length *jn; or, without a list, the
// one window's buckets 0 .. B-1, whole): CTAs that stride over the items (queue == nullptr) or
// persistent CTAs that take items from a device work queue (an atomic counter)
// until it runs dry.  Buckets of radix windows are joined through direct
// tables when their key indices allow it.
//
// A persistent CTA works one item ahead: while it joins item k, item k+1's
// record is already in shared memory and its two runs are being prefetched
// into L2, and item k+2's record is on its way (an asynchronous copy into
// shared memory, from the index claimed during item k-1).  So no step of a
// bucket waits on the queue, the list or the first loads of its runs.
// kModels: the call has learned buckets (and no raw windows).
// A CTA's place in the grid when the items are too few for two per SM: the first
// CTAs of the SMs in front, in the order in which they ask, the others from the
// end back.  A grid of two CTAs per SM does not come to the SMs quite in turn:
// the second CTAs of some are started before the first of others, and with their
// buckets these end last (128 buckets of 16,384 tuples per side: 604 us a call by
// position, 519 so).  n, zeroed: first ones, others, CTAs seen on each SM.
constexpr uint32_t kSpreadSms = 256;
constexpr size_t kQueueBytes = 32 + sizeof(uint32_t) * (2 + kSpreadSms) + 8;   // the queues, then n (whole 16 bytes)
static_assert(kQueueBytes % 16 == 0, "the heavy sums follow");
__device__ __noinline__ uint32_t spread_cta(uint32_t *n) {
    uint32_t sm;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
    if (atomicAdd(&n[2 + sm % kSpreadSms], 1u) == 0) return atomicAdd(&n[0], 1u);
    return gridDim.x - 1 - atomicAdd(&n[1], 1u);
}

template <bool kModels>
__global__ void __launch_bounds__(kJoinThreads, 2)
bucket_join_count_kernel(const sjbg_tuple *__restrict__ L, const sjbg_tuple *__restrict__ R,
                         const WinPlan *__restrict__ wins, uint64_t *__restrict__ partL,
                         uint64_t *__restrict__ partR, const uint32_t *__restrict__ start,
                         const uint32_t *__restrict__ cnt, uint32_t B, WinAcc *__restrict__ acc, uint32_t cap,
                         uint32_t *queue, const JoinItem *__restrict__ items, const uint32_t *__restrict__ jn,
                         const RowsJoin rj) {
    if (kModels && rj.queue) rows_join(rj, wins, acc, cap);   // ends with a barrier
    const uint32_t nitems = items ? *jn : B;
    uint32_t clean = 0, turn = 0;
    auto join = [&](const JoinItem &ji) {
        if (ji.nB == 0 || ji.nP == 0) return;
        const JoinRuns jr = join_runs(ji, L, R, wins, partL, partR);
        if (ji.flags & kItemHot) {
            join_count_hot(static_cast<const uint64_t *>(jr.b), ji.nB, static_cast<const uint64_t *>(jr.p), ji.nP,
                           jr.bside, &acc[ji.w], cap);
            clean = 0;
            return;
        }
        unsigned long long count = 0, prod = 0;
        if constexpr (!kModels) {
            if (ji.flags & kItemRaw) {
                join_item<true, kModels>(ji, jr, cap, clean, turn, count, prod);
                flush_acc(&acc[ji.w], count, 0, prod);
                return;
            }
        }
        join_item<false, kModels>(ji, jr, cap, clean, turn, count, prod);
        flush_acc(&acc[ji.w], count, 0, prod);
    };
    if (!queue || !items) {
        for (uint32_t i = blockIdx.x; items && i < nitems; i += gridDim.x) {
            SJBG_BARRIER();   // the previous item's shared-memory readers are done
            join(items[i]);
        }
        if (items || blockIdx.x >= nitems) return;
        JoinItem ji;
        {
            const uint32_t i = blockIdx.x, nL = cnt[i], nR = cnt[B + i];
            const bool swap = nR < nL;
            ji.nB = swap ? nR : nL; ji.nP = swap ? nL : nR;
            ji.sB = swap ? start[B + i] : start[i]; ji.sP = swap ? start[i] : start[B + i];
            ji.w = 0; ji.lg = wins[0].log2_buckets; ji.flags = swap ? kItemSwap : 0u; ji.pad = 0;
        }
        join(ji);
        return;
    }
    __shared__ JoinItem slot_s[3];   // item k, k+1, k+2 (by position: cur_s, then the two ahead)
    __shared__ uint32_t cur_s, valid_s;   // slot of item k; bit q: slot (cur + q) % 3 holds an item
    uint32_t claim = 0;                   // thread 0: index claimed for item k+2
    if (threadIdx.x == 0) {
        // the first two items are the CTA's by its place; the queue hands out the rest
        const uint32_t i0 = nitems <= gridDim.x / 2 ? spread_cta(queue + 8) : blockIdx.x, i1 = gridDim.x + blockIdx.x;
        claim = 2 * gridDim.x + atomicAdd(queue, 1u);
        if (i0 < nitems) slot_s[0] = items[i0];
        if (i1 < nitems) slot_s[1] = items[i1];
        cur_s = 0;
        valid_s = (i0 < nitems ? 1u : 0u) | (i1 < nitems ? 2u : 0u);
    }
    SJBG_BARRIER();
    while (valid_s & 1u) {
        const uint32_t c = cur_s, v = valid_s;
        // learned calls read the record in shared memory as they go (z = 0.5, 2 x 4 M:
        // 76 us with it in registers, 74 without); for the others it is the other way
        // round (2 x 2^24 dense tuples: 129 and 139)
        using Item = std::conditional_t<kModels, const JoinItem &, const JoinItem>;
        Item ji = slot_s[c];
        const uint32_t c1 = c == 2 ? 0u : c + 1u, c2 = c1 == 2 ? 0u : c1 + 1u;
        uint32_t claim_next = 0;
        if (threadIdx.x == 0) {
            if (v & 2u) {   // item k+1: its runs into L2 while item k is joined
                const JoinItem nx = slot_s[c1];
                const JoinRuns nr = join_runs(nx, L, R, wins, partL, partR);
                const size_t word = (nx.flags & kItemRaw) ? sizeof(sjbg_tuple) : sizeof(uint64_t);
                l2_prefetch_bulk(nr.b, word * nx.nB);
                l2_prefetch_bulk(nr.p, word * nx.nP);
            }
            if (claim < nitems) {   // item k+2's record: shared memory, without blocking
                const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&slot_s[c2]);
                const JoinItem *src = items + claim;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n"
                             "cp.async.cg.shared.global [%2], [%3], 16;\n"
                             "cp.async.commit_group;\n" ::"r"(dst), "l"(src), "r"(dst + 16u),
                             "l"(reinterpret_cast<const uint8_t *>(src) + 16)
                             : "memory");
            }
            claim_next = 2 * gridDim.x + atomicAdd(queue, 1u);   // read after this item's join
        }
        join(ji);
        if (threadIdx.x == 0) {
            asm volatile("cp.async.wait_all;\n" ::: "memory");
            cur_s = c1;
            valid_s = (v >> 1) | (claim < nitems ? 2u : 0u);
            claim = claim_next;
        }
        SJBG_BARRIER();
    }
}

// ---- calls of unpartitioned windows only
// Small windows are all launches: the general path's upload, clears, scan,
// join and result copy took 28 us on the device for one window of 4,096 tuples
// per side, of which the tuples are well under one.  Here the host lists the
// items, the one kernel gets them by value (or reads them in pinned memory),
// and its last CTA writes the results to pinned memory, leaving its
// accumulators zero for the next call.  Windows beyond one table are cut on
// both sides while the pieces make one wave of CTAs: the work grows with their
// product, but one window of 65,536 tuples per side is done in 24 us on the
// device, where partitioning it first takes 28 and an HBM table 30.
struct RawItem {
    uint64_t b, p;   // first build and probe tuple, in their sides' arrays
    uint32_t nB, nP, w, flags;
};
constexpr uint32_t kRawByValue = 64;
struct RawItems {
    RawItem v[kRawByValue];
};
constexpr uint32_t kRawWindows = 1024;   // accumulators kept

// Matches of the windows of raw-only calls, and the CTAs that are done.
struct RawAcc {
    unsigned long long count[kRawWindows], prod[kRawWindows];
    uint32_t done;
};

__global__ void __launch_bounds__(kJoinThreads, 2)
raw_join_kernel(const sjbg_tuple *__restrict__ L, const sjbg_tuple *__restrict__ R,
                const __grid_constant__ RawItems items, const RawItem *__restrict__ list, uint32_t n, uint32_t cap,
                RawAcc *__restrict__ acc, WinAcc *__restrict__ out) {
    __shared__ unsigned long long part[2][kJoinThreads / 32];
    __shared__ uint32_t last_s;
    const RawItem it = list ? list[blockIdx.x] : items.v[blockIdx.x];
    const bool swap = (it.flags & kItemSwap) != 0;
    JoinItem ji;
    ji.nB = it.nB; ji.nP = it.nP; ji.sB = 0; ji.sP = 0;
    ji.w = it.w; ji.lg = 0; ji.flags = it.flags; ji.pad = 0;
    JoinRuns jr;
    jr.b = const_cast<sjbg_tuple *>((swap ? R : L) + it.b);   // (never written)
    jr.p = (swap ? L : R) + it.p;
    jr.bside = swap ? 1u : 0u;
    uint32_t clean = 0, turn = 0;
    unsigned long long count = 0, prod = 0;
    if (it.nB && it.nP) join_item<true, false>(ji, jr, cap, clean, turn, count, prod);
    count = warp_sum_u64(count);
    prod = warp_sum_u64(prod);
    if (lane_id() == 0) {
        part[0][warp_id()] = count;
        part[1][warp_id()] = prod;
    }
    SJBG_BARRIER();
    if (threadIdx.x == 0) {
        for (uint32_t q = 1; q < kJoinThreads / 32; q++) {
            count += part[0][q];
            prod += part[1][q];
        }
        if (gridDim.x == 1) {
            last_s = 2;
        } else {
            if (count) atomicAdd(&acc->count[it.w], count);
            if (prod) atomicAdd(&acc->prod[it.w], prod);
            __threadfence();
            last_s = atomicAdd(&acc->done, 1u) == gridDim.x - 1 ? 1u : 0u;
            __threadfence();
        }
    }
    SJBG_BARRIER();
    if (last_s == 0) return;
    for (uint32_t w = threadIdx.x; w <= n; w += kJoinThreads) {   // out[n]: the call's status word
        WinAcc r{0, 0, 0, 0, 0};
        if (last_s == 2) {
            if (w == it.w) {   // (thread it.w holds no sum: thread 0's are in part)
                for (uint32_t q = 0; q < kJoinThreads / 32; q++) {
                    r.count += part[0][q];
                    r.prod += part[1][q];
                }
            }
        } else if (w < n) {
            r.count = atomicExch(&acc->count[w], 0ull);
            r.prod = atomicExch(&acc->prod[w], 0ull);
        }
        out[w] = r;
    }
    if (last_s == 1 && threadIdx.x == 0) acc->done = 0;
}

// One CTA per join item (the grid covers the longest possible list).
__global__ void __launch_bounds__(kJoinThreads)
bucket_join_enum_kernel(const uint64_t *__restrict__ partL, const uint64_t *__restrict__ partR,
                        WinAcc *__restrict__ acc, const WinPlan *__restrict__ wins, sjbg_pair *__restrict__ pairs,
                        uint32_t table_bits, const JoinItem *__restrict__ items, const uint32_t *__restrict__ jn) {
    if (blockIdx.x < *jn) join_enum_bucket(items[blockIdx.x], partL, partR, acc, wins, pairs, table_bits);
}

// ------------------------------------------------------------------ host driver
static uint32_t ceil_log2(uint64_t x) {
    uint32_t b = 0;
    while (((uint64_t)1 << b) < x) b++;
    return b;
}

// The partitioner of a call: the configured one, or for SJBG_PART_AUTO the
// autotuner's choice, else one HBM table per window when every window's table
// stays well inside L2 (at most 2^18 left tuples, 2^21 over the call), else
// radix partitioning.
uint32_t choose_partitioner(const sjbg_handle *h, const WinHost *wins, uint32_t n) {
    if (h->cfg.partitioner != SJBG_PART_AUTO) return h->cfg.partitioner;
    if (h->tune.partitioner) return h->tune.partitioner;
    uint64_t tot = 0, mx = 0;
    for (uint32_t w = 0; w < n; w++) {
        tot += wins[w].n_left;
        mx = std::max(mx, wins[w].n_left);
    }
    return (mx <= (1u << 18) && tot <= (1u << 21)) ? SJBG_PART_NONE : SJBG_PART_RADIX;
}

// Slots of a count table for buckets of the target size (a target whose table
// would not fit is joined in passes).
static uint32_t join_cap(const sjbg_handle *h, uint64_t target) {
    return (uint32_t)std::min<size_t>(count_table_cap((uint32_t)target),
                                      (h->max_smem_optin - count_table_bytes(0) - 1024) / 16);
}

int hj_raw_batch(sjbg_handle *h, const sjbg_tuple *dL, const sjbg_tuple *dR, const WinHost *wins, uint32_t n,
                 WinAcc *hAcc, bool *done) {
    *done = false;
    if (h->cfg.partitioner != SJBG_PART_AUTO || (h->tune.partitioner && h->tune.partitioner != SJBG_PART_NONE) ||
        n == 0 || n > kRawWindows)
        return SJBG_OK;
    const uint32_t cap = join_cap(h, h->tune.bucket_target);
    const uint64_t slots = 2 * (uint64_t)std::max(h->num_sms, 1);   // resident CTAs
    uint64_t tuples = 0;
    bool small = true;   // every build side fits one table
    for (uint32_t w = 0; w < n; w++) {
        const uint64_t nB = std::min(wins[w].n_left, wins[w].n_right), nP = std::max(wins[w].n_left, wins[w].n_right);
        if (nP > 0xFFFFFFFFull) return SJBG_OK;
        small &= nB < cap;
        tuples += nB + nP;
    }
    // Any cut of the two runs will do (the sums are over pairs of tuples).  The
    // smallest square pieces that make one wave of CTAs; windows that need more
    // are taken when every build side fits a table, whole build sides with pieces of
    // the probes that cost the SMs about equal shares.  (With the build sides cut to
    // a share too, every probe piece met several: 32 windows of 20,000 and 5,000
    // tuples 85 us instead of 35, 2 of 500,000 and 5,000 94 instead of 39.)
    uint32_t piece = 0, chunk = 0;
    for (uint32_t s = kRawPiece; s <= kRawPieceMost && s < cap && piece == 0; s += kRawPiece / 2) {
        uint64_t items = 0;
        for (uint32_t w = 0; w < n && items <= slots; w++)
            items += ((wins[w].n_left + s - 1) / s) * ((wins[w].n_right + s - 1) / s);
        if (items <= slots) piece = chunk = s;
    }
    if (piece == 0) {
        if (!small) return SJBG_OK;
        const uint64_t share = tuples / (2 * slots);
        piece = cap - 1;
        chunk = (uint32_t)std::min<uint64_t>(kJoinChunk, std::max<uint64_t>(kRawPiece, share));
    }
    std::vector<RawItem> list;
    for (uint32_t w = 0; w < n; w++) {
        const WinHost &x = wins[w];
        if (!x.n_left || !x.n_right) continue;
        const bool swap = x.n_right < x.n_left;
        const uint32_t nB = (uint32_t)(swap ? x.n_right : x.n_left), nP = (uint32_t)(swap ? x.n_left : x.n_right);
        const uint64_t b0 = swap ? x.right_off : x.left_off, p0 = swap ? x.left_off : x.right_off;
        const uint32_t kb = (nB + piece - 1) / piece, per = std::max(chunk, nB / kb);
        const uint32_t kp = (uint32_t)(((uint64_t)nP + per - 1) / per);
        for (uint32_t i = 0; i < kb; i++)
            for (uint32_t j = 0; j < kp; j++) {
                const uint32_t b = (uint32_t)((uint64_t)nB * i / kb), p = (uint32_t)((uint64_t)nP * j / kp);
                list.push_back(RawItem{b0 + b, p0 + p, (uint32_t)((uint64_t)nB * (i + 1) / kb) - b,
                                       (uint32_t)((uint64_t)nP * (j + 1) / kp) - p, w,
                                       kItemRaw | (swap ? (uint32_t)kItemSwap : 0u)});
            }
    }
    if (list.empty()) {   // nothing can match
        std::memset(hAcc, 0, sizeof(WinAcc) * (n + 1));
        *done = true;
        return SJBG_OK;
    }
    const bool fresh = h->ws[WS_RAW_ACC].p == nullptr;
    RawAcc *acc = static_cast<RawAcc *>(ws_get(h, WS_RAW_ACC, sizeof(RawAcc)));
    if (!acc) return fail(h, SJBG_E_NOMEM, "window accumulators");
    if (fresh) SJBG_CK(h, cudaMemsetAsync(acc, 0, sizeof(RawAcc), h->stream));
    RawItems items;
    const RawItem *dList = nullptr;
    if (list.size() <= kRawByValue) {
        std::copy(list.begin(), list.end(), items.v);
    } else {
        RawItem *hst = static_cast<RawItem *>(pinned_get(h, 0, sizeof(RawItem) * list.size()));
        if (!hst) return fail(h, SJBG_E_NOMEM, "plan buffers");
        std::copy(list.begin(), list.end(), hst);
        dList = hst;
    }
    const size_t smem = std::max({count_table_bytes(cap), kDirectBytes, kPlaceBytes});
    allow_big_smem(raw_join_kernel, smem);
    SJBG_CK(h, launch(h, "raw_join", raw_join_kernel, dim3((uint32_t)list.size()), dim3(kJoinThreads), smem, dL, dR,
                      items, dList, n, cap, acc, hAcc));
    *done = true;
    return SJBG_OK;
}

int hj_lazy_batch(sjbg_handle *h, const sjbg_tuple *dL, const sjbg_tuple *dR, const WinHost *wins, uint32_t n,
                  sjbg_pair *dPairs, WinAcc *acc, bool enumerate, uint32_t *part_used) {
    if (n == 0) return SJBG_OK;
    const uint32_t part = choose_partitioner(h, wins, n);
    if (part == SJBG_PART_NONE) {   // one HBM table per window (hj_global.cu)
        if (part_used) *part_used = SJBG_PART_NONE;
        return hj_global_batch(h, dL, dR, wins, n, dPairs, acc, enumerate);
    }
    const bool learned = part == SJBG_PART_LEARNED;
    if (part_used) *part_used = learned ? SJBG_PART_LEARNED : SJBG_PART_RADIX;
    // build tuples per bucket: 2048 when chains are built, else the tuned target
    const uint64_t target = enumerate ? 2048 : h->tune.bucket_target;
    const uint32_t cap = join_cap(h, target);

    // ---- plan
    std::vector<WinPlan> plan(n);
    std::vector<uint32_t> tileL(n + 1), tileR(n + 1), hgL(n + 1), hgR(n + 1), itL(n + 1), itR(n + 1);
    std::vector<uint32_t> pbL(n + 1), pbR(n + 1);   // window bases in the partitioned arrays
    uint64_t B = 0, totL = 0, totR = 0;
    uint32_t maxP = 1, rows_lg = 0;   // rows_lg: log2 of the most buckets of a window joined from sorted tiles
    // a learned window may be joined from sorted tiles; with a table near the shared
    // memory's size (large bucket targets) there is no room for their lists
    const bool rows_fit = learned && !enumerate && rows_join_bytes(cap) + 1024 <= h->max_smem_optin;
    bool any_two = false, any_one = false, any_raw = false;
    for (uint32_t w = 0; w < n; w++) {
        const WinHost &wh = wins[w];
        WinPlan &p = plan[w];
        p.left_off = wh.left_off; p.n_left = wh.n_left; p.right_off = wh.right_off; p.n_right = wh.n_right;
        p.pairs_off = wh.pairs_off; p.pairs_cap = dPairs ? wh.pairs_cap : 0;
        // a counting join builds from the smaller side of a bucket, so the fan-out
        // follows the window's smaller side
        const uint64_t build = enumerate ? wh.n_left : std::min(wh.n_left, wh.n_right);
        uint32_t lg;
        if (learned) lg = learned_log2_buckets(h, wh.n_left);
        else if (h->cfg.radix_bits) lg = h->cfg.radix_bits;
        else lg = ceil_log2((build + target - 1) / target);
        lg = std::min(lg, kMaxBucketsLog2);
        if (wh.n_left == 0 || wh.n_right == 0) lg = 0;
        // (a handle that names radix partitioning gets it for every window; the join
        // of a learned call, which a tuned automatic handle may make, takes none)
        p.raw = h->cfg.partitioner == SJBG_PART_AUTO && !learned && !enumerate && lg == 0 && build < cap ? 1u : 0u;
        p.log2_buckets = lg;
        p.bucket_base = (uint32_t)B;
        p.model = 0xFFFFFFFFu;
        p.two_level = lg >= kTwoLevelMinLog2 ? 1u : 0u;
        any_two |= p.two_level != 0;
        any_one |= p.two_level == 0 && !p.raw;
        any_raw |= p.raw != 0;
        B += 1ull << lg;
        maxP = std::max(maxP, 1u << lg);
        // (no tile of an unpartitioned window is counted or scattered)
        tileL[w + 1] = tileL[w] + (p.raw ? 0u : (uint32_t)((wh.n_left + kTile - 1) / kTile));
        tileR[w + 1] = tileR[w] + (p.raw ? 0u : (uint32_t)((wh.n_right + kTile - 1) / kTile));
        p.rows = rows_fit && lg > 0 ? 1u : 0u;
        if (p.rows) rows_lg = std::max(rows_lg, std::min(lg, kRowsMaxLog2));
        // fine-pass CTAs: coarse partitions x groups of kGroupTiles tiles
        const uint32_t nc = 1u << coarse_bits(lg);
        itL[w + 1] = itL[w] + nc * ((tileL[w + 1] - tileL[w] + kGroupTiles - 1) / kGroupTiles);
        itR[w + 1] = itR[w] + nc * ((tileR[w + 1] - tileR[w] + kGroupTiles - 1) / kGroupTiles);
        totL += wh.n_left;
        totR += wh.n_right;
        pbL[w + 1] = (uint32_t)std::min<uint64_t>(totL, 0xFFFFFFFFull);
        pbR[w + 1] = (uint32_t)std::min<uint64_t>(totR, 0xFFFFFFFFull);
    }
    if (B > 0xFFFFFFFFull / 4 || totL >= 0xFFFFFFFFull || totR >= 0xFFFFFFFFull)
        return fail(h, SJBG_E_CAPACITY, "hash join batch exceeds 2^32 tuples per side");
    // counting CTAs per window side: shares of about T / (resident CTAs) tiles,
    // so that one wave holds the call when its window sides are large and the
    // set-up of each CTA is paid over many tiles.  A share has at least
    // kHistTiles tiles with a model (whose copy and heavy-key sums each CTA sets
    // up), and for radix windows at least as many as make flushing the P
    // counters cheap (2, or P / 256, up to kHistTiles): a call of few tiles
    // otherwise leaves most SMs idle (one window of 2^20 tuples per side, 490
    // tiles: 32 CTAs of 16 tiles took 17.5 us; 2^21 per side in 2^14 buckets, 16
    // CTAs of 64 tiles 156 us, 64 of 16 50).
    // When many sides are smaller than a share (uneven batches), shares of an
    // eighth of that keep the CTAs small enough to balance the SMs.
    uint32_t join_chunk;
    {
        const size_t histSmem = sizeof(uint32_t) * ((maxP + 1) / 2 * 2) + sizeof(uint64_t) * kTile;
        allow_big_smem(part_hist_kernel, histSmem);
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, part_hist_kernel, kPartThreads, histSmem) !=
            cudaSuccess)
            return fail(h, SJBG_E_CUDA, "counting pass occupancy");
        const uint64_t slots = (uint64_t)std::max(per_sm, 1) * (uint64_t)std::max(h->num_sms, 1);
        const uint64_t T = (uint64_t)tileL[n] + tileR[n];
        const uint64_t least = learned ? kHistTiles : std::min<uint64_t>(kHistTiles, std::max<uint64_t>(2, maxP / 256));
        uint64_t share = std::max<uint64_t>(least, (T + slots - 1) / slots);
        uint64_t ctas = 0;
        for (uint32_t w = 0; w < n; w++)
            ctas += (tileL[w + 1] - tileL[w] + share - 1) / share + (tileR[w + 1] - tileR[w] + share - 1) / share;
        if (ctas > slots + slots / 8) share = std::max<uint64_t>(least, T / (8 * slots));
        for (uint32_t w = 0; w < n; w++) {
            hgL[w + 1] = hgL[w] + (uint32_t)((tileL[w + 1] - tileL[w] + share - 1) / share);
            hgR[w + 1] = hgR[w] + (uint32_t)((tileR[w + 1] - tileR[w] + share - 1) / share);
        }
        // probe tuples per join piece: small enough to spread a call over the SMs, at most kJoinChunk
        // (chains cost more to build: with pieces of 4,000 probes the enumerating
        // join of 500,009 and 2,000,003 tuples took 78 us, against 66)
        join_chunk = (uint32_t)std::min<uint64_t>(
            kJoinChunk, std::max<uint64_t>(enumerate ? kJoinChunkEnum : kJoinChunkMin,
                                           (totL + totR) / (4 * (uint64_t)std::max(h->num_sms, 1))));
    }
    // (two CTAs per SM)
    const uint32_t hot_unit = (uint32_t)std::max<uint64_t>(1, (totL + totR) / (kHotFactor * 2 * (uint64_t)std::max(h->num_sms, 1)));
    const uint64_t max_items = join_items_bound(B, totL + totR, join_chunk, enumerate ? 0x0FFFFFFFu : cap);
    if (max_items > 0x7FFFFFFFull) return fail(h, SJBG_E_CAPACITY, "hash join batch has too many join items");

    // ---- upload plan, tile prefixes and (learned) the
    // sampling plan in one copy
    const size_t planB = sizeof(WinPlan) * n, tileB = sizeof(uint32_t) * (n + 1);
    const size_t lsOff = (planB + 8 * tileB + 15) & ~(size_t)15;
    const size_t upB = lsOff + (learned ? learned_stage_bytes(n) : 0);
    uint8_t *hst = static_cast<uint8_t *>(pinned_get(h, 0, upB));
    uint8_t *dev = static_cast<uint8_t *>(ws_get(h, WS_WIN_PLAN, upB));
    if (!hst || !dev) return fail(h, SJBG_E_NOMEM, "plan buffers");
    std::memcpy(hst, plan.data(), planB);
    std::memcpy(hst + planB, tileL.data(), tileB);
    std::memcpy(hst + planB + tileB, tileR.data(), tileB);
    std::memcpy(hst + planB + 2 * tileB, hgL.data(), tileB);
    std::memcpy(hst + planB + 3 * tileB, hgR.data(), tileB);
    std::memcpy(hst + planB + 4 * tileB, itL.data(), tileB);
    std::memcpy(hst + planB + 5 * tileB, itR.data(), tileB);
    std::memcpy(hst + planB + 6 * tileB, pbL.data(), tileB);
    std::memcpy(hst + planB + 7 * tileB, pbR.data(), tileB);
    LearnedStage lst{};
    if (learned) lst = learned_stage(h, plan.data(), n, hst + lsOff);
    // what starts from zero is zeroed by the same launch as the upload, with no
    // clears between the kernels later: the bucket counters; per window side its
    // compacted light tuples, then the join list's length; the join's queues
    // (join items, then, 16 bytes on, the buckets joined from sorted tiles) and the
    // join CTAs' places; the heavy keys' sums
    const size_t ccntOff = sizeof(uint32_t) * 2 * B;
    const size_t queueOff = (ccntOff + sizeof(uint32_t) * (2 * n + 1) + 15) & ~(size_t)15, heavyOff = queueOff + kQueueBytes;
    const size_t zeroB = heavyOff + (learned ? sizeof(HeavyAcc) * kMaxHeavy * n : 0);
    uint8_t *dZero = static_cast<uint8_t *>(ws_get(h, WS_BUCKET_CNT, zeroB));
    if (!dZero) return fail(h, SJBG_E_NOMEM, "partition buffers");
    if (int rc_up = stage_copy_zero(h, dev, hst, upB, dZero, zeroB)) return rc_up;
    uint32_t *dCnt = reinterpret_cast<uint32_t *>(dZero);
    uint32_t *dCcnt = reinterpret_cast<uint32_t *>(dZero + ccntOff);
    uint32_t *queues = reinterpret_cast<uint32_t *>(dZero + queueOff);
    HeavyAcc *dHeavy = learned ? reinterpret_cast<HeavyAcc *>(dZero + heavyOff) : nullptr;
    WinPlan *dPlan = reinterpret_cast<WinPlan *>(dev);
    const uint32_t *dTileL = reinterpret_cast<const uint32_t *>(dev + planB);
    const uint32_t *dTileR = reinterpret_cast<const uint32_t *>(dev + planB + tileB);
    const uint32_t *dHgL = reinterpret_cast<const uint32_t *>(dev + planB + 2 * tileB);
    const uint32_t *dHgR = reinterpret_cast<const uint32_t *>(dev + planB + 3 * tileB);
    const uint32_t *dItL = reinterpret_cast<const uint32_t *>(dev + planB + 4 * tileB);
    const uint32_t *dItR = reinterpret_cast<const uint32_t *>(dev + planB + 5 * tileB);
    const uint32_t *dPbL = reinterpret_cast<const uint32_t *>(dev + planB + 6 * tileB);
    const uint32_t *dPbR = reinterpret_cast<const uint32_t *>(dev + planB + 7 * tileB);

    uint32_t *dStart = static_cast<uint32_t *>(ws_get(h, WS_BUCKET_START, sizeof(uint32_t) * 2 * B));
    uint32_t *dCur = static_cast<uint32_t *>(ws_get(h, WS_BUCKET_CURSOR, sizeof(uint32_t) * 2 * B));
    uint64_t *dPL = static_cast<uint64_t *>(ws_get(h, WS_PART_LEFT, sizeof(uint64_t) * std::max<uint64_t>(totL, 1)));
    uint64_t *dPR = static_cast<uint64_t *>(ws_get(h, WS_PART_RIGHT, sizeof(uint64_t) * std::max<uint64_t>(totR, 1)));
    if (!dStart || !dCur || !dPL || !dPR) return fail(h, SJBG_E_NOMEM, "partition buffers");

    const LearnedModel *dModels = nullptr;
    if (learned) {
        int rc = learned_prepare(h, dL, dR, lst, dev + lsOff, n, dPlan, &dModels, !enumerate);
        if (rc) return rc;
    }
    // the counting pass's output: per window side and tile, its light tuples
    // (compacted windows: packed at the side's start; others: sorted by coarse
    // partition inside the tile's own region), plus the tiles' coarse rows
    const uint64_t tiles64 = (uint64_t)tileL[n] + tileR[n];
    uint64_t *dComp = static_cast<uint64_t *>(ws_get(h, WS_COMPACT, sizeof(uint64_t) * kTile * std::max<uint64_t>(tiles64, 1)));
    uint32_t *dRows = static_cast<uint32_t *>(ws_get(h, WS_COARSE_ROWS, sizeof(uint32_t) * kRow * std::max<uint64_t>(tiles64, 1)));
    uint32_t *dJn = dCcnt + 2 * n;
    // the passes' work prefixes (kWorkArrays of n + 1), then (16-byte aligned) the join list
    const size_t workWords = (kWorkArrays * (size_t)(n + 1) + 3) & ~(size_t)3;
    uint32_t *dWork = static_cast<uint32_t *>(
        ws_get(h, WS_TILE_PREFIX, sizeof(uint32_t) * workWords + sizeof(JoinItem) * (size_t)max_items));
    JoinItem *dJlist = dWork ? reinterpret_cast<JoinItem *>(dWork + workWords) : nullptr;
    // sorted tiles' rows
    const uint32_t rstride = sorted_row(1u << rows_lg);
    uint16_t *dRows16 = nullptr;
    if (rows_lg) {
        dRows16 = static_cast<uint16_t *>(ws_get(h, WS_ROWS16, sizeof(uint16_t) * rstride * std::max<uint64_t>(tiles64, 1)));
        if (!dRows16) return fail(h, SJBG_E_NOMEM, "partition staging buffers");
    }
    if (!dComp || !dRows || !dWork) return fail(h, SJBG_E_NOMEM, "partition staging buffers");
    uint64_t *dCompR = dComp + (uint64_t)kTile * tileL[n];

    const uint32_t tiles = tileL[n] + tileR[n];
    auto scan = [&]() {
        return launch(h, "part_scan", part_scan_win_kernel, dim3(n), dim3(1024), 0, (const WinPlan *)dPlan, dPbL, dPbR,
                      (const uint32_t *)dCnt, dStart, dCur, (uint32_t)B, dModels, dJlist, dJn, join_chunk,
                      enumerate ? 0x0FFFFFFFu : cap, hot_unit, !enumerate, (const uint32_t *)dCcnt);
    };
    if (!tiles && any_raw) SJBG_CK(h, scan());
    if (tiles) {
        const size_t histSmem = sizeof(uint32_t) * ((maxP + 1) / 2 * 2) + sizeof(uint64_t) * kTile;
        SJBG_CK(h, launch(h, "part_hist", part_hist_kernel, dim3(hgL[n] + hgR[n]), dim3(kPartThreads), histSmem, dL,
                          dR, dPlan, n, dTileL, dTileR, dHgL, dHgR, dCnt, (uint32_t)B, dModels, dHeavy, dComp, dCompR,
                          dCcnt, dRows));
        if (learned)
            SJBG_CK(h, launch(h, "heavy_finish", heavy_finish_kernel, dim3(n), dim3(256), 0, (const WinPlan *)dPlan, n,
                              dModels, (const HeavyAcc *)dHeavy, acc));
        // the tiles each later pass has work for (compacted windows: their light tiles only)
        SJBG_CK(h, launch(h, "part_work", part_work_kernel, dim3(1), dim3(32 * kWorkArrays), 0, (const WinPlan *)dPlan, n, dTileL,
                          dTileR, dItL, dItR, dModels, (const uint32_t *)dCcnt, dWork));
        if (learned && !enumerate) {   // compacted windows exist only with heavy keys
            const size_t lightSmem = kTile * sizeof(uint64_t) + sizeof(uint32_t) * maxP;
            allow_big_smem(part_light_kernel, lightSmem);
            SJBG_CK(h, launch(h, "part_light", part_light_kernel, dim3(std::min<uint32_t>(tiles, 2u * (uint32_t)h->num_sms)),
                              dim3(kPartThreads), lightSmem, (const WinPlan *)dPlan, n, dTileL, dTileR,
                              (const uint32_t *)dWork, dCnt, (uint32_t)B, dModels, dComp, dCompR, (const uint32_t *)dCcnt,
                              dRows16, rstride));
        }
        SJBG_CK(h, scan());
        // single-level windows, and compacted windows (their packed light tuples):
        // a local counting sort per tile
        if (any_one || (learned && !enumerate)) {
            const size_t scatterSmem = kTile * (sizeof(uint64_t) + sizeof(uint16_t)) + 2 * sizeof(uint32_t) * maxP;
            // without a learned partitioner every window is radix-partitioned
            auto scatter = learned ? part_scatter_kernel<false> : part_scatter_kernel<true>;
            allow_big_smem(scatter, scatterSmem);
            // (radix runs of neighbours: 1,024 windows 3,415 us with 3 CTAs per SM, 3,380
            // with 6, 3,350 with 12, 3,324 with 24)
            const uint32_t sgrid = std::min<uint32_t>(tiles, 3u * (learned ? 4u : 8u) * (uint32_t)h->num_sms);
            const uint32_t *wS = dWork + 2 * kWorkScatter * (n + 1);
            SJBG_CK(h, launch(h, "part_scatter", scatter, dim3(sgrid), dim3(kPartThreads), scatterSmem,
                              dL, dR, dPlan, n, dTileL, dTileR, wS, wS + (n + 1), dCur, (uint32_t)B, dPL, dPR,
                              dModels, (const uint64_t *)dComp, (const uint64_t *)dCompR, (const uint32_t *)dCcnt));
        }
        // two-level windows: the fine pass over the tiles' coarse runs
        if (any_two && itL[n] + itR[n]) {
            allow_big_smem(part_fine_kernel, kFineSmem);
            const uint32_t fgrid = std::min<uint32_t>(itL[n] + itR[n], 4u * 4u * (uint32_t)h->num_sms);
            SJBG_CK(h, launch(h, "part_fine", part_fine_kernel, dim3(fgrid), dim3(kFineThreads), kFineSmem,
                              (const WinPlan *)dPlan, n, dTileL, dTileR, (const uint32_t *)dWork, dCur, (uint32_t)B,
                              dPL, dPR, dModels, (const uint64_t *)dComp, (const uint64_t *)dCompR,
                              (const uint32_t *)dRows));
        }
    }
    // persistent CTAs draining a work queue of join items, or about one CTA per item
    uint32_t *queue = nullptr;
    dim3 jgrid((uint32_t)std::min<uint64_t>(max_items, B + (totL + totR) / join_chunk));
    if (enumerate) {   // (chain-building joins: one CTA per item)
        const uint32_t bits = 13;   // 8192 slots for chunks of 4096
        const size_t smem = sizeof(uint32_t) * (2 * ((1u << bits) + 1) + 2 * kEnumChunk);
        allow_big_smem(bucket_join_enum_kernel, smem);
        SJBG_CK(h, launch(h, "bucket_join_enum", bucket_join_enum_kernel, jgrid, dim3(kJoinThreads), smem,
                          (const uint64_t *)dPL, (const uint64_t *)dPR, acc, (const WinPlan *)dPlan, dPairs, bits,
                          (const JoinItem *)dJlist, (const uint32_t *)dJn));
    } else {
        const size_t smem = std::max({count_table_bytes(cap), kDirectBytes, kPlaceBytes, rows_lg ? rows_join_bytes(cap) : 0});
        RowsJoin rj{};
        if (rows_lg && tiles)
            rj = RowsJoin{n, rstride, dTileL, dTileR, (const uint32_t *)dWork, (const uint32_t *)dCcnt,
                          dComp, dCompR, (const uint16_t *)dRows16, queues + 4};
        auto join = learned ? bucket_join_count_kernel<true> : bucket_join_count_kernel<false>;
        allow_big_smem(join, smem);
        if (h->tune.persistent_join && max_items > (uint64_t)h->num_sms) {
            queue = queues;
            // as many persistent CTAs as fit on an SM at this table size (at most 2 by registers)
            const uint32_t per_sm = std::max<uint32_t>(1, (uint32_t)((228u << 10) / (smem + 1024)));
            jgrid = dim3((uint32_t)std::min<uint64_t>(max_items, (uint64_t)h->num_sms * std::min<uint32_t>(per_sm, 2u)));
        }
        SJBG_CK(h, launch(h, "bucket_join_count", join, jgrid, dim3(kJoinThreads), smem, dL, dR,
                          (const WinPlan *)dPlan, dPL, dPR, (const uint32_t *)dStart, (const uint32_t *)dCnt,
                          (uint32_t)B, acc, cap, queue, (const JoinItem *)dJlist, (const uint32_t *)dJn, rj));
    }
    return SJBG_OK;
}


// ------------------------------------------------------------------ caller-provided scratch
// One window, count mode, radix partitioning, every buffer carved out of the
// caller-provided device scratch `sc` (no allocation, no host-to-device copy:
// the plan is written by a set-up kernel).  Used by the allocation-free entry
// point in noalloc.cu.
struct RawScratch {
    WinPlan plan;
    uint32_t tile[8];   // tileL {0, tL}, tileR {0, tR}, hgL {0, gL}, hgR {0, gR}
    WinAcc acc[2];      // the window's accumulator, then the call's device status word (acc[1].info, kErr* bits)
};

// Byte offsets of the scratch buffers from a 256-byte aligned base: the
// RawScratch record, the bucket arrays (counts, starts and cursors, 2P words
// each) and the partitioned sides (8 bytes per tuple).  The
// size check of the entry point and the carving below both use it.
struct RawLayout {
    size_t rs, cnt, part_left, part_right, end;
};

static size_t round256(size_t b) { return (b + 255) & ~size_t(255); }

static RawLayout raw_layout(uint64_t nL, uint64_t nR, uint32_t P) {
    RawLayout l;
    l.rs = 0;
    l.cnt = round256(sizeof(RawScratch));
    l.part_left = l.cnt + round256(sizeof(uint32_t) * 6 * (size_t)P);
    l.part_right = l.part_left + sizeof(uint64_t) * std::max<uint64_t>(nL, 1);
    l.end = l.part_right + sizeof(uint64_t) * std::max<uint64_t>(nR, 1);
    return l;
}

// Radix fan-out of a window: about 4,096 left tuples per bucket; one bucket when a side is empty.
static uint32_t raw_log2_buckets(uint64_t nL, uint64_t nR) {
    uint32_t lg = 0;
    while (((uint64_t)4096 << lg) < nL) lg++;
    return (nL == 0 || nR == 0) ? 0 : lg;
}

__global__ void raw_setup_kernel(RawScratch *rs, uint32_t *cnt, uint32_t P, uint64_t nL, uint64_t nR, uint32_t lg,
                                 uint32_t tL, uint32_t tR) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        WinPlan &p = rs->plan;
        p.left_off = 0; p.n_left = nL; p.right_off = 0; p.n_right = nR;
        p.pairs_off = 0; p.pairs_cap = 0;
        p.bucket_base = 0; p.log2_buckets = lg; p.model = 0xFFFFFFFFu; p.two_level = 0; p.raw = 0; p.rows = 0;
        rs->tile[0] = 0; rs->tile[1] = tL;
        rs->tile[2] = 0; rs->tile[3] = tR;
        rs->tile[4] = 0; rs->tile[5] = (tL + kHistTiles - 1) / kHistTiles;
        rs->tile[6] = 0; rs->tile[7] = (tR + kHistTiles - 1) / kHistTiles;
        rs->acc[0] = WinAcc{0, 0, 0, 0, 0};
        rs->acc[1] = WinAcc{0, 0, 0, 0, 0};
    }
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < 2 * P; i += gridDim.x * blockDim.x) cnt[i] = 0;
}

// The window's result, with the device status word turned into a status code
// (the bits the batched path maps in device_status_error).
__global__ void raw_finish_kernel(const RawScratch *rs, sjbg_window_result *out) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        const unsigned long long bits = rs->acc[1].info;
        sjbg_window_result r;
        r.count = rs->acc[0].count;
        r.xor_checksum = 0;
        r.prod_checksum = rs->acc[0].prod;
        r.n_pairs = 0;
        r.status = !bits ? SJBG_OK
                         : (bits & kErrTimeout) ? SJBG_E_TIMEOUT
                                                : SJBG_E_CAPACITY;   // a table or queue could not take its input
        r.flags = 0;
        r.partitioner_used = SJBG_PART_RADIX;
        r.ms = 0.0f;
        *out = r;
    }
}

size_t hj_raw_scratch_bytes(uint64_t max_tuples) {
    const uint32_t P = 1u << raw_log2_buckets(max_tuples, max_tuples);
    return 255 + raw_layout(max_tuples, max_tuples, P).end;   // 255: aligning the caller's base
}

static uint8_t *align256(uint8_t *p) { return reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(p) + 255) & ~uintptr_t(255)); }

int hj_count_window_raw(const sjbg_tuple *dL, uint64_t nL, const sjbg_tuple *dR, uint64_t nR, uint8_t *sc,
                        size_t sc_bytes, sjbg_window_result *dOut, cudaStream_t st) {
    const uint32_t lg = raw_log2_buckets(nL, nR);
    const uint32_t P = 1u << lg;
    const uint32_t tL = (uint32_t)((nL + kTile - 1) / kTile), tR = (uint32_t)((nR + kTile - 1) / kTile);
    uint8_t *base = align256(sc);
    const RawLayout lay = raw_layout(nL, nR, P);
    if (base + lay.end > sc + sc_bytes)
        return fail(nullptr, SJBG_E_CAPACITY, "sjbg_lazy_hj_noalloc: the window does not fit the fixed scratch");
    RawScratch *rs = reinterpret_cast<RawScratch *>(base + lay.rs);
    uint32_t *cnt = reinterpret_cast<uint32_t *>(base + lay.cnt);
    uint32_t *start = cnt + 2 * P;
    uint32_t *cur = start + 2 * P;
    uint64_t *pL = reinterpret_cast<uint64_t *>(base + lay.part_left);
    uint64_t *pR = reinterpret_cast<uint64_t *>(base + lay.part_right);
    // an error left pending by the caller's own earlier work is not this call's
    cudaGetLastError();
    auto launched = [](const char *what) -> int {
        const cudaError_t e = cudaGetLastError();
        return e == cudaSuccess ? SJBG_OK : cuda_fail(nullptr, e, what);
    };
    raw_setup_kernel<<<4, 256, 0, st>>>(rs, cnt, P, nL, nR, lg, tL, tR);
    if (int rc = launched("sjbg_lazy_hj_noalloc: raw_setup_kernel")) return rc;
    const uint32_t *tl = rs->tile;
    if (tL && tR) {
        const uint32_t groups = (tL + kHistTiles - 1) / kHistTiles + (tR + kHistTiles - 1) / kHistTiles;
        allow_big_smem(part_hist_kernel, sizeof(uint32_t) * P);
        part_hist_kernel<<<groups, kPartThreads, sizeof(uint32_t) * P, st>>>(
            dL, dR, &rs->plan, 1, tl, tl + 2, tl + 4, tl + 6, cnt, P, nullptr, nullptr, nullptr, nullptr, nullptr,
            nullptr);
        if (int rc = launched("sjbg_lazy_hj_noalloc: part_hist_kernel")) return rc;
        part_scan_kernel<<<1, 1024, 0, st>>>(cnt, start, cur, P);
        if (int rc = launched("sjbg_lazy_hj_noalloc: part_scan_kernel")) return rc;
        const size_t scatterSmem = kTile * (sizeof(uint64_t) + sizeof(uint16_t)) + 2 * sizeof(uint32_t) * P;
        allow_big_smem(part_scatter_kernel<true>, scatterSmem);
        // a single-level radix window: the scatter work is every tile
        part_scatter_kernel<true><<<tL + tR, kPartThreads, scatterSmem, st>>>(dL, dR, &rs->plan, 1, tl, tl + 2, tl, tl + 2,
                                                                          cur, P, pL, pR, nullptr, nullptr, nullptr,
                                                                          nullptr);
        if (int rc = launched("sjbg_lazy_hj_noalloc: part_scatter_kernel")) return rc;
        const uint32_t cap = count_table_cap(4096);
        const size_t smem = std::max({count_table_bytes(cap), kDirectBytes, kPlaceBytes});
        allow_big_smem(bucket_join_count_kernel<false>, smem);
        bucket_join_count_kernel<false><<<P, kJoinThreads, smem, st>>>(dL, dR, &rs->plan, pL, pR, start, cnt, P, rs->acc,
                                                                cap, nullptr, nullptr, nullptr, RowsJoin{});
        if (int rc = launched("sjbg_lazy_hj_noalloc: bucket_join_count_kernel")) return rc;
    }
    raw_finish_kernel<<<1, 32, 0, st>>>(rs, dOut);
    return launched("sjbg_lazy_hj_noalloc: raw_finish_kernel");
}

}  // namespace sjbg
