// trtc_segmented.cuh -- batched segmented sort + scan: many independent segments of one
// key/value array, each stably sorted by key and then exclusive-scanned (Plus) over its
// sorted values, in one persistent launch fed by a device work queue.
//
// The reference sorts one vector per call (internal/radix_sort.cpp:165-553) and scans one
// vector per call (internal/general_scan.cpp:8-88); a batch there is one call pair per
// segment.  Here a CTA takes a segment id from the queue and sorts the whole segment itself,
// in one of six size classes (ITEMS and warp_small are the tuning table's; launch_segmented.cu):
//   * segments of at most `warp_small` (0 or 32) keys: one warp, a bitonic network over
//     (code, index) pairs, no digit counters (seg_warp_bitonic);
//   * segments of at most 32 * ITEMS keys: one warp, 8-bit LSD passes of ballot
//     ranking (two or three by the top varying bits and a fix-up of ties, SegPlan, else all) with per-warp counters (seg_warp_sort_scan); a CTA's eight warps take eight
//     such segments at once;
//   * segments of at most 64 * ITEMS / 128 * ITEMS keys: a group of two / four warps, the
//     same passes with the group's counters scanned by the group and named barriers of the
//     group only (seg_group_sort_scan); a CTA's four / two groups take as many segments;
//   * small segments (<= 256 * ITEMS keys) are sorted on chip: the same passes of
//     warp multisplit ranking + shared-memory scatter, with the tile re-laid out so that
//     every warp gets keys whatever the segment length; then the values are scanned and
//     keys, values and scan are written once;
//   * larger segments: from two tiles up one stable scatter pass through the temp array cuts
//     the segment into up to 256 buckets by its top varying bits, and the bucket counts carry
//     the value sums that start each bucket's scan; the CTA's warps, then groups of warps, then
//     the whole CTA sort and scan the buckets on chip.  Shorter ones, and segments with a
//     bucket above a tile, take LSD passes in global memory: one read builds all digit
//     histograms, chunked, stable scatter passes ping-pong between the segment and the temp
//     array (mostly L2-resident for segments of up to a few MB), then a chunked scan with a
//     running carry.
// The queue lists the segments by class, largest first, so the longest work starts first and
// a CTA's batch of small segments shares one class.
#pragma once
#include "trtc_prelude.cuh"
#include "trtc_radix.cuh"

namespace trtc {

// One segment given by its own arrays (list mode, used by the request server): keys k and
// 4-byte values v sorted in place, out = exclusive scan of the sorted values (or nullptr),
// n elements, toff = the segment's offset in the temp arrays.
struct SegItem {
    void* k;
    void* v;
    void* out;
    unsigned long long n;
    unsigned long long toff;
};

// size classes of a segment of `len` keys (items = keys per thread of a CTA tile): 0 one
// warp, 1 / 2 two / four warps, 3 the CTA on chip, 4 + k the CTA through global memory with
// floor(log2 len) = floor(log2 (256 items)) + k.  The work queue lists the classes from the
// largest down, so the longest segments start first.
enum { SEG_CLASSES = 32 };
TRTC_FORCEINLINE uint32_t seg_class(unsigned long long len, uint32_t items) {
    const unsigned long long tile = 256ull * items;
    if (len > tile) {
        const int k = (63 - __clzll((long long)len)) - (63 - __clzll((long long)tile));
        return 4u + (uint32_t)min(k, SEG_CLASSES - 5);
    }
    return len > 128ull * items ? 3u : len > 64ull * items ? 2u : len > 32ull * items ? 1u : 0u;
}

struct SegCtrl {
    unsigned long long next;                   // work-queue cursor
    unsigned long long count[SEG_CLASSES];     // segments per class
    unsigned long long placed[SEG_CLASSES];    // segments of a class placed so far
    unsigned long long pad;
};

// per-class segment counts (block histogram, one atomic per class and block)
template <class OFF>
__global__ void __launch_bounds__(256) seg_class_count_kernel(const OFF* __restrict__ off, unsigned long long nseg,
                                                              uint32_t items, SegCtrl* ctrl) {
    __shared__ unsigned long long s_c[SEG_CLASSES];
    if (threadIdx.x < SEG_CLASSES) s_c[threadIdx.x] = 0;
    __syncthreads();
    for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < nseg;
         i += (unsigned long long)gridDim.x * blockDim.x)
        atomicAdd(&s_c[seg_class((unsigned long long)(off[i + 1] - off[i]), items)], 1ull);
    __syncthreads();
    if (threadIdx.x < SEG_CLASSES && s_c[threadIdx.x]) atomicAdd(&ctrl->count[threadIdx.x], s_c[threadIdx.x]);
}

// queue[] = the segments ordered by class, largest class first (order inside a class is free).
// A CTA reserves the places of its 256 segments with one atomic per class: one per segment
// serialised on the few class words (100k segments: 66 us for the count and this kernel, now 21).
template <class OFF>
__global__ void __launch_bounds__(256) seg_queue_kernel(const OFF* __restrict__ off, unsigned long long nseg,
                                                        uint32_t items, uint32_t* __restrict__ queue, SegCtrl* ctrl) {
    __shared__ unsigned long long s_start[SEG_CLASSES], s_base[SEG_CLASSES];
    __shared__ uint32_t s_n[SEG_CLASSES];
    if (threadIdx.x == 0) {
        unsigned long long run = 0;
        for (int c = SEG_CLASSES - 1; c >= 0; c--) { s_start[c] = run; run += ctrl->count[c]; }
    }
    for (unsigned long long b = (unsigned long long)blockIdx.x * blockDim.x; b < nseg;
         b += (unsigned long long)gridDim.x * blockDim.x) {
        if (threadIdx.x < SEG_CLASSES) s_n[threadIdx.x] = 0;
        __syncthreads();
        const unsigned long long i = b + threadIdx.x;
        uint32_t c = 0, r = 0;
        if (i < nseg) {
            c = seg_class((unsigned long long)(off[i + 1] - off[i]), items);
            r = atomicAdd(&s_n[c], 1u);
        }
        __syncthreads();
        if (threadIdx.x < SEG_CLASSES && s_n[threadIdx.x])
            s_base[threadIdx.x] = s_start[threadIdx.x] + atomicAdd(&ctrl->placed[threadIdx.x], (unsigned long long)s_n[threadIdx.x]);
        __syncthreads();
        if (i < nseg) queue[s_base[c] + r] = (uint32_t)i;
        __syncthreads();
    }
}

// ------------------------------------------------------------------ which digits a segment needs
// A segment of n keys is told apart by far fewer bits than its keys have: the top 16 of the
// bits that vary in it leave n^2 / 2^17 pairs of uniform keys tied (0.5 of a pair at n = 256,
// 32 at 2048).  So a segment is sorted by those bits only, two 8-bit passes, or by the top 24,
// three, and the short runs of tied keys that are left are finished in place by the thread at
// each run's first key (stable: a key only passes larger ones).  Bits above the highest
// varying one take no pass in either form.
struct SegPlan {
    uint32_t shift;   // the passes sort the codes' bits shift .. shift + 8 passes - 1
    uint32_t passes;
    // of a form that may take two passes: the ties left by three are copies of one another, most likely
    TRTC_FORCEINLINE bool copies(uint32_t q0) const { return q0 == 2u && passes == 3u; }
};

template <class K> constexpr uint32_t seg_min_passes() {
    return is_same<K, float>::value || is_same<K, double>::value ? 3u : 2u;
}

// Longest run of tied keys finished in place on chip, and the work spent on one in global memory, in keys
// read and moved.  A longer one that is out of order sends the segment to the passes over all its
// varying bits (any order the short form leaves keeps equal keys in input order, so they start
// from there).
enum { SEG_RUN = 16, SEG_STEPS_FAR = 512, SEG_FIXED = 1, SEG_LONG = 2, SEG_DUPS = 3 };

template <class K> constexpr uint32_t seg_dups3() { return sizeof(typename RadixKey<K>::U) == 4 ? 128u : ~0u; }

// the key's ordered code, descending order folded in
template <class K, bool DESC>
TRTC_FORCEINLINE typename RadixKey<K>::U seg_code(typename RadixKey<K>::B k) {
    typedef typename RadixKey<K>::U U;
    const U u = RadixKey<K>::ordered(k);
    return DESC ? (U)~u : u;
}

template <class K, bool DESC>
TRTC_FORCEINLINE uint32_t seg_digit(typename RadixKey<K>::B k, uint32_t shift) {
    return (uint32_t)(seg_code<K, DESC>(k) >> shift) & 0xFFu;
}

// OR over the warp
template <class U>
TRTC_FORCEINLINE U seg_warp_or(U x) {
    if constexpr (sizeof(U) == 8) {
        const uint32_t lo = __reduce_or_sync(0xffffffffu, (uint32_t)x);
        const uint32_t hi = __reduce_or_sync(0xffffffffu, (uint32_t)((unsigned long long)x >> 32));
        return (U)(((unsigned long long)hi << 32) | lo);
    } else {
        return (U)__reduce_or_sync(0xffffffffu, (uint32_t)x);
    }
}

// true when two of the warp's sampled codes (`in` lanes) agree above `shift` and differ below:
// 1 in 130 samples of 32 uniform keys at 16 bits, nearly every one of clustered keys.  With `dups`
// also when SEG_DUPS of them are copies of others: keys with so many copies (fewer than 170
// equally likely values, or a few popular ones) leave long runs at any shift.
template <class U>
__device__ inline bool seg_sample_ties(U code, bool in, uint32_t shift, bool dups) {
    bool tie = false, copy = false;
    const uint32_t m = __ballot_sync(0xffffffffu, in);
    if (in) {
        const uint32_t peers = __match_any_sync(m, code >> shift);
        const U first = __shfl_sync(m, code, (int)__ffs(peers) - 1);
        tie = first != code;
        copy = !tie && (peers & lanemask_lt()) != 0u;
    }
    return __any_sync(0xffffffffu, tie) || (dups && __popc(__ballot_sync(0xffffffffu, copy)) >= (int)SEG_DUPS);
}

// all varying bits: `diff` has a bit set where two keys of the segment differ
template <class U>
TRTC_FORCEINLINE SegPlan seg_full_plan(U diff) {
    const uint32_t bits = diff ? 64u - (uint32_t)__clzll((long long)(unsigned long long)diff) : 1u;
    return {0u, (bits + 7u) / 8u};
}

// the short form of at least `q0` passes where it saves one, leaves less than one tied key in
// four for uniform keys and `ties(shift, dups)` does not show clustered ones; else all varying bits.
// q0 is 2 on chip, 3 in global memory, where a tie costs several round trips (2^24 u32 keys in
// segments of 10,000: 891 us with two passes, 694 with three, 722 with all four), and 3 for
// floats: sign, exponent and 7 bits of the mantissa tie most keys of a few hundred (2^24 normal
// floats in segments of 2000: 754 us with two where the samples allow it, 538 with three).
// B200, 2^24 keys in equal segments, all digits -> this plan, us: u32 of 64 keys 1384 -> 894,
// 250 570 -> 363, 500 438 -> 289, 2000 500 -> 412; i64 3659 -> 1263, 1388 -> 529, 1067 -> 397,
// 1072 -> 573; f32 2054 -> 1789, 757 -> 649, 585 -> 499, 548 -> 538.  What bounds it is the
// instruction rate of the ranking (eight ballots and an atomic per key and pass).
// Segments of more than 128 keys of which many are copies (SEG_DUPS) take no two-pass form: one other key
// in a long run of copies costs all passes again, which eight more bits make rare.  4-byte keys take all
// digits then (`dups3`): the question whether the runs are in order costs their kernel 2 to 3 % where there
// are none, more than a pass saved in segments of copies is worth.  B200, 2^24 keys in segments of 250 / 1000 /
// 2000, us, all digits by the former passes, the short form for every segment, this rule: u32 of 64 values
// 555 / 516 / 483, 526 / 659 / 623, 524 / 545 / 543; u32 ids of a Zipf(1.1) popularity 558 / 518 / 485, 504 / 578 /
// 569, 531 / 545 / 545; f32 of 64 values 761 / 597 / 546, 865 / 925 / 842, 728 / 635 / 605; i64 of 64 values 1362 /
// 1117 / 1046, 759 / 942 / 901, 627 / 608 / 631; i64 ids in segments of 80,000 2113, 4592, 2184.
template <class U, class TIES>
__device__ inline SegPlan seg_plan(U diff, uint32_t len, uint32_t q0, uint32_t dups3, TIES ties) {
    const uint32_t dups2 = 128u;
    const uint32_t bits = diff ? 64u - (uint32_t)__clzll((long long)(unsigned long long)diff) : 1u;
    for (uint32_t q = q0; q <= 3; q++)
        if (8u * q < bits && len <= (1u << (8u * q - 2u)) && !ties(bits - 8u * q, len > (q < 3u ? dups2 : dups3)))
            return {bits - 8u * q, q};
    return seg_full_plan(diff);
}

// Element e of a segment that is sorted by its bits from `shift` up: if it is the first of a
// run of tied keys, insertion-sorts the run's first SEG_RUN keys, or as far as SEG_STEPS_FAR go (FAR).  The tied bits of a slot do
// not change while other threads sort their runs, so the neighbours may be read meanwhile.
template <class K, class V, bool DESC, bool FAR>
__device__ inline uint32_t seg_fix_run(volatile typename RadixKey<K>::B* sk, V* sv, uint32_t e, uint32_t len,
                                       uint32_t shift) {
    typedef typename RadixKey<K>::B KB;
    typedef typename RadixKey<K>::U U;
    if (e + 1 >= len) return 0u;
    const U pre = seg_code<K, DESC>(sk[e]) >> shift;
    if ((seg_code<K, DESC>(sk[e + 1]) >> shift) != pre) return 0u;
    if (e > 0 && (seg_code<K, DESC>(sk[e - 1]) >> shift) == pre) return 0u;
    uint32_t steps = 0;
    for (uint32_t j = e + 1; j < len; j++) {
        const KB kj = sk[j];
        const U cj = seg_code<K, DESC>(kj);
        if ((cj >> shift) != pre) break;
        if (FAR ? ++steps > (uint32_t)SEG_STEPS_FAR : j - e >= (uint32_t)SEG_RUN) return (uint32_t)SEG_FIXED | (uint32_t)SEG_LONG;
        uint32_t i = j;
        if (seg_code<K, DESC>(sk[i - 1]) <= cj) continue;
        const V vj = sv[j];
        do {
            sk[i] = sk[i - 1];
            sv[i] = sv[i - 1];
            i--;
            if (FAR) steps++;
        } while (i > e && seg_code<K, DESC>(sk[i - 1]) > cj);
        sk[i] = kj;
        sv[i] = vj;
    }
    return (uint32_t)SEG_FIXED;
}

// seg_fix_run for the elements first, first + stride, ... below end: the ties are collected
// for 32 of them before the first run is sorted, so the lanes of a warp sort their runs at the
// same time (row by row nearly every row of 32 has one lane with a run)
template <class K, class V, bool DESC>
__device__ inline uint32_t seg_fix_runs(typename RadixKey<K>::B* sk, V* sv, uint32_t first, uint32_t stride,
                                        uint32_t end, uint32_t len, uint32_t shift) {
    const uint32_t last = min(end, len - 1u);  // the segment's last key starts no run
    uint32_t fixed = 0;
    for (; first < last; first += 32u * stride) {
        uint32_t mask = 0;
#pragma unroll 4
        for (uint32_t r = 0; r < 32u; r++) {
            const uint32_t e = first + r * stride;
            if (e >= last) break;
            const bool tie = ((seg_code<K, DESC>(sk[e]) ^ seg_code<K, DESC>(sk[e + 1])) >> shift) == 0;
            mask |= tie ? 1u << r : 0u;
        }
        while (mask) {
            const uint32_t e = first + (uint32_t)(__ffs((int)mask) - 1) * stride;
            mask &= mask - 1u;
            fixed |= seg_fix_run<K, V, DESC, false>(sk, sv, e, len, shift);
        }
    }
    return fixed;
}

// Is any of the ties among these elements out of order?  (Copies are not: where a plan expects them, nobody
// looks into the runs of a segment without an inverted tie.)
template <class K, bool DESC>
__device__ inline bool seg_ties_inverted(const typename RadixKey<K>::B* sk, uint32_t first, uint32_t stride, uint32_t end,
                                         uint32_t len, uint32_t shift) {
    typedef typename RadixKey<K>::U U;
    const uint32_t last = min(end, len - 1u);
    bool inv = false;
#pragma unroll 4
    for (; first < last; first += stride) {
        const U a = seg_code<K, DESC>(sk[first]), b = seg_code<K, DESC>(sk[first + 1]);
        inv |= ((a ^ b) >> shift) == 0 && a > b;
    }
    return inv;
}

// true where element e is smaller than the one before it
template <class K, bool DESC>
TRTC_FORCEINLINE bool seg_inverted(const volatile typename RadixKey<K>::B* sk, uint32_t e) {
    return e > 0 && seg_code<K, DESC>(sk[e - 1]) > seg_code<K, DESC>(sk[e]);
}

// Ranks IT (<= ITEMS) warp-striped items per thread of a tile of `tile_n` keys: element
// e = warp*32*IT + i*32 + lane.  On return pos[i] is the item's position in the digit-sorted
// tile (stable), s_cnt[d] / s_start[d] the tile's digit counts and exclusive starts.
template <class K, bool DESC, int ITEMS>
__device__ inline void seg_rank_tile(const typename RadixKey<K>::B (&keys)[ITEMS], uint32_t (&pos)[ITEMS], int IT,
                                     uint32_t tile_n, uint32_t shift, uint32_t* s_whist, uint32_t* s_cnt,
                                     uint32_t* s_start, uint32_t* s_wsum) {
    constexpr int WARPS = 8;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < WARPS * 256; i += 256) s_whist[i] = 0;
    __syncthreads();
    uint32_t* wh = s_whist + warp * 256;
    const uint32_t ltm = lanemask_lt();
    const uint32_t wbase = warp * 32u * (uint32_t)IT;
    uint32_t info[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
        pos[i] = 0;
        info[i] = 0;
        if (i >= IT || wbase + (uint32_t)i * 32u >= tile_n) continue;  // warp-uniform
        const bool valid = wbase + (uint32_t)i * 32u + lane < tile_n;
        const uint32_t d = seg_digit<K, DESC>(keys[i], shift);
        uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
        for (int b = 0; b < 8; b++) {
            const bool set = (d >> b) & 1u;
            const uint32_t bb = __ballot_sync(0xffffffffu, set);
            peers &= set ? bb : ~bb;
        }
        const uint32_t leader = 31u - __clz(peers);
        info[i] = (uint32_t)__popc(peers & ltm) | (leader << 8);
        if (valid && lane == leader) pos[i] = atomicAdd(&wh[d], (uint32_t)__popc(peers));
    }
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
        if (i >= IT || wbase + (uint32_t)i * 32u >= tile_n) continue;
        pos[i] = __shfl_sync(0xffffffffu, pos[i], (int)(info[i] >> 8)) + (info[i] & 0xFFu);
    }
    __syncthreads();
    const uint32_t d = threadIdx.x;
    uint32_t cnt = 0;
#pragma unroll
    for (int w = 0; w < WARPS; w++) cnt += s_whist[w * 256 + d];
    const uint32_t start = block_excl_scan_256<256>(cnt, s_wsum);
    s_cnt[d] = cnt;
    s_start[d] = start;
    uint32_t run = start;
#pragma unroll
    for (int w = 0; w < WARPS; w++) {
        const uint32_t c = s_whist[w * 256 + d];
        s_whist[w * 256 + d] = run;
        run += c;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
        if (i >= IT || wbase + (uint32_t)i * 32u + lane >= tile_n) continue;
        pos[i] += wh[seg_digit<K, DESC>(keys[i], shift)];
    }
}

// exclusive Plus scan of s_v[0..len) into s_o (256 threads, len <= 256 * ITEMS), carry-in c
template <class V, int ITEMS>
__device__ inline V seg_block_excl_scan(const V* s_v, V* s_o, uint32_t len, V carry, V* s_part) {
    const uint32_t t = threadIdx.x;
    const uint32_t per = (len + 255u) / 256u;  // consecutive elements per thread
    const uint32_t b = t * per;
    V sum = V();
    for (uint32_t k = 0; k < per; k++)
        if (b + k < len) sum += s_v[b + k];
    // block exclusive scan of the thread sums (values of any width: two warp levels)
    const uint32_t lane = t & 31u, w = t >> 5;
    V x = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const V y = shfl_up_any(x, d);
        if (lane >= (uint32_t)d) x += y;
    }
    if (lane == 31) s_part[w] = x;
    __syncthreads();
    V pre = carry;
    for (uint32_t i = 0; i < w; i++) pre += s_part[i];
    V total = carry;
    for (int i = 0; i < 8; i++) total += s_part[i];
    V run = pre + x - sum;
    for (uint32_t k = 0; k < per; k++)
        if (b + k < len) { s_o[b + k] = run; run += s_v[b + k]; }
    __syncthreads();
    return total;
}

// One warp sorts (stable LSD, 8-bit digits) and scans a segment of len <= 32 * ITEMS keys on
// its own: no block barrier, so the CTA's eight warps work on eight small segments at once.
// Element e = i*32 + lane sits in item i of the lane; sk / sv are this warp's staging slices
// (32 * ITEMS elements), wh its 256 digit counters.  ik / iv: where the keys and values are read
// (gk / gv for a segment in place); carry: the scan's first value.
template <class K, class V, bool DESC, int ITEMS>
__device__ inline void seg_warp_sort_scan(const typename RadixKey<K>::B* ik, const V* iv, typename RadixKey<K>::B* gk,
                                          V* gv, V* gs, uint32_t len, V carry, typename RadixKey<K>::B* sk, V* sv,
                                          uint32_t* wh) {
    typedef typename RadixKey<K>::B KB;
    typedef typename RadixKey<K>::U U;
    constexpr uint32_t Q0 = seg_min_passes<K>();
    const uint32_t lane = threadIdx.x & 31u;
    const int IT = (int)((len + 31u) / 32u);  // items in use (warp-uniform)
    const uint32_t ltm = lanemask_lt();
    KB k[ITEMS];
    V v[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
        const uint32_t e = (uint32_t)i * 32u + lane;
        if (i < IT && e < len) { k[i] = ik[e]; v[i] = iv[e]; }
        else { k[i] = KB(0); v[i] = V(); }
    }
    const U ref = seg_code<K, DESC>(ik[0]);
    U diff = 0;
#pragma unroll
    for (int i = 0; i < ITEMS; i++)
        if (i < IT && (uint32_t)i * 32u + lane < len) diff |= seg_code<K, DESC>(k[i]) ^ ref;
    diff = seg_warp_or(diff);
    SegPlan plan = seg_plan(diff, len, Q0, seg_dups3<K>(), [&](uint32_t sh, bool dups) {
        return seg_sample_ties(seg_code<K, DESC>(k[0]), lane < len, sh, dups);
    });
    uint32_t shift = plan.shift;
    for (uint32_t p = 0; p < plan.passes; p++) {
#pragma unroll
        for (int j = 0; j < 8; j++) wh[j * 32 + lane] = 0;
        __syncwarp();
        uint32_t pos[ITEMS], info[ITEMS];
#pragma unroll
        for (int i = 0; i < ITEMS; i++) {
            pos[i] = 0;
            info[i] = 0;
            if (i >= IT) continue;
            const bool valid = (uint32_t)i * 32u + lane < len;
            const uint32_t d = seg_digit<K, DESC>(k[i], shift);
            uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
            for (int b = 0; b < 8; b++) {
                const bool set = (d >> b) & 1u;
                const uint32_t bb = __ballot_sync(0xffffffffu, set);
                peers &= set ? bb : ~bb;
            }
            const uint32_t leader = 31u - __clz(peers | 1u);
            info[i] = (uint32_t)__popc(peers & ltm) | (leader << 8);
            if (valid && lane == leader) pos[i] = atomicAdd(&wh[d], (uint32_t)__popc(peers));
        }
#pragma unroll
        for (int i = 0; i < ITEMS; i++)
            if (i < IT) pos[i] = __shfl_sync(0xffffffffu, pos[i], (int)(info[i] >> 8)) + (info[i] & 0xFFu);
        __syncwarp();
        // exclusive scan of the 256 counters: lane owns digits 8*lane .. 8*lane+7
        uint32_t c[8], sum = 0;
#pragma unroll
        for (int j = 0; j < 8; j++) { c[j] = wh[lane * 8 + j]; sum += c[j]; }
        uint32_t inc = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, d);
            if (lane >= (uint32_t)d) inc += y;
        }
        uint32_t run = inc - sum;
#pragma unroll
        for (int j = 0; j < 8; j++) { wh[lane * 8 + j] = run; run += c[j]; }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < ITEMS; i++) {
            if (i >= IT || (uint32_t)i * 32u + lane >= len) continue;
            const uint32_t q = pos[i] + wh[seg_digit<K, DESC>(k[i], shift)];
            sk[q] = k[i];
            sv[q] = v[i];
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < ITEMS; i++) {
            const uint32_t e = (uint32_t)i * 32u + lane;
            if (i < IT && e < len) { k[i] = sk[e]; v[i] = sv[e]; }
        }
        __syncwarp();
        shift += 8u;
        if (p + 1 < plan.passes || plan.shift == 0) continue;
        // the last pass of the short form: the runs of tied keys
        if constexpr (sizeof(U) == 8 || Q0 == 3u)
            if ((Q0 == 3u || plan.copies(Q0)) &&
                !__any_sync(0xffffffffu, seg_ties_inverted<K, DESC>(sk, lane, 32u, len, len, plan.shift)))
                continue;
        const uint32_t fixed =
            __reduce_or_sync(0xffffffffu, seg_fix_runs<K, V, DESC>(sk, sv, lane, 32u, len, len, plan.shift));
        __syncwarp();
        if (fixed) {
#pragma unroll
            for (int i = 0; i < ITEMS; i++) {
                const uint32_t e = (uint32_t)i * 32u + lane;
                if (i < IT && e < len) { k[i] = sk[e]; v[i] = sv[e]; }
            }
        }
        if (fixed & (uint32_t)SEG_LONG) {
            bool inv = false;
            for (uint32_t e = lane; e < len; e += 32u) inv |= seg_inverted<K, DESC>(sk, e);
            if (__any_sync(0xffffffffu, inv)) {
                plan = seg_full_plan(diff);
                shift = 0;
                p = ~0u;  // from the first pass again
            }
        }
        __syncwarp();
    }
    // exclusive scan of the sorted values, written with the sorted keys and values
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
        if (i >= IT) continue;
        const uint32_t e = (uint32_t)i * 32u + lane;
        const bool valid = e < len;
        const V x = valid ? v[i] : V();
        V incl = x;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const V y = shfl_up_any(incl, d);
            if (lane >= (uint32_t)d) incl += y;
        }
        if (valid) {
            gk[e] = k[i];
            gv[e] = v[i];
            if (gs) gs[e] = carry + incl - x;
        }
        carry += shfl_any(incl, 31);
    }
}

// A group of G (2 or 4) warps sorts (stable LSD, 8-bit digits) and scans a segment of
// len <= 32 * G * ITEMS keys: the segment is cut into G consecutive warp chunks of 32 * IT
// elements (element e = wg*32*IT + i*32 + lane in item i of lane `lane` of the group's warp
// wg, IT = ceil(len / (32 G))); each warp ranks its chunk with ballots and its own 256 digit
// counters, the group scans the counters digit-major / warp-minor (so equal digits keep the
// chunk order), and the keys are scattered to the group's staging slice sk.  The values are
// not held in registers: they move between the group's two value slices va / vb (element e
// read from the current one, written to its new slot in the other).  Only the group's warps
// meet at its named barrier `bar` (1 + group index, 32 * G threads), so the CTA's 8 / G
// groups work on 8 / G segments at once.  s_wsum / s_vpart: one slot per warp of the CTA.
template <class K, class V, bool DESC, int ITEMS>
__device__ __noinline__ void seg_group_sort_scan(const typename RadixKey<K>::B* ik, const V* iv,
                                                 typename RadixKey<K>::B* gk, V* gv, V* gs, uint32_t len, V carry,
                                                 typename RadixKey<K>::B* sk, V* va, V* vb, uint32_t* s_whist,
                                                 uint32_t* s_wsum, V* s_vpart, uint32_t G, uint32_t bar) {
    // G is a runtime value (2 or 4): one copy of this code serves both group sizes, which
    // keeps the kernel inside its register budget
    typedef typename RadixKey<K>::B KB;
    typedef typename RadixKey<K>::U U;
    constexpr uint32_t Q0 = seg_min_passes<K>();
    const uint32_t GT = 32u * G;      // threads of the group
    const uint32_t DPT = 256u / GT;   // digits scanned per thread
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t wg = warp % G, gw0 = warp - wg;  // warp inside the group, the group's first warp
    const uint32_t gt = wg * 32u + lane;             // thread inside the group
    const uint32_t IT = (len + GT - 1u) / GT;        // items in use (group-uniform)
    const uint32_t wbase = wg * 32u * IT;
    const uint32_t wn = len > wbase ? min(len - wbase, 32u * IT) : 0u;  // elements of this warp
    uint32_t* wh = s_whist + warp * 256;
    const uint32_t ltm = lanemask_lt();
    // named barrier of the group (immediate ids, so the kernel reserves barriers 0-4 only)
    auto gsync = [&]() {
        switch (bar) {
            case 1: asm volatile("bar.sync 1, %0;\n" ::"r"(GT) : "memory"); break;
            case 2: asm volatile("bar.sync 2, %0;\n" ::"r"(GT) : "memory"); break;
            case 3: asm volatile("bar.sync 3, %0;\n" ::"r"(GT) : "memory"); break;
            default: asm volatile("bar.sync 4, %0;\n" ::"r"(GT) : "memory"); break;
        }
    };
    KB k[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
        const uint32_t r = (uint32_t)i * 32u + lane;
        if ((uint32_t)i < IT && r < wn) { k[i] = ik[wbase + r]; va[wbase + r] = iv[wbase + r]; }
        else k[i] = KB(0);
    }
    const U ref = seg_code<K, DESC>(ik[0]);
    U diff = 0;
#pragma unroll
    for (int i = 0; i < ITEMS; i++)
        if ((uint32_t)i < IT && (uint32_t)i * 32u + lane < wn) diff |= seg_code<K, DESC>(k[i]) ^ ref;
    diff = seg_warp_or(diff);
    if (lane == 0) {
        wh[0] = (uint32_t)diff;
        wh[1] = (uint32_t)((unsigned long long)diff >> 32);
    }
    gsync();
    for (uint32_t w = 0; w < G; w++) {
        const uint32_t* cw = &s_whist[(gw0 + w) * 256];
        diff |= (U)(((unsigned long long)cw[1] << 32) | cw[0]);
    }
    // (every warp looks at the same G samples, spread over the segment)
    SegPlan plan = seg_plan(diff, len, Q0, seg_dups3<K>(), [&](uint32_t sh, bool dups) {
        bool tie = false;
        for (uint32_t w = 0; w < G; w++)
            tie |= seg_sample_ties(seg_code<K, DESC>(ik[(len / GT) * (w * 32u + lane)]), true, sh, dups);
        return tie;
    });
    gsync();  // the counters are free
    uint32_t shift = plan.shift;
    for (uint32_t p = 0; p < plan.passes; p++) {
#pragma unroll
        for (int j = 0; j < 8; j++) wh[j * 32 + lane] = 0;
        __syncwarp();
        uint32_t pos[ITEMS];
#pragma unroll
        for (int i = 0; i < ITEMS; i++) {
            pos[i] = 0;
            if ((uint32_t)i >= IT || (uint32_t)i * 32u >= wn) continue;  // warp-uniform
            const bool valid = (uint32_t)i * 32u + lane < wn;
            const uint32_t d = seg_digit<K, DESC>(k[i], shift);
            uint32_t peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
            for (int b = 0; b < 8; b++) {
                const bool set = (d >> b) & 1u;
                const uint32_t bb = __ballot_sync(0xffffffffu, set);
                peers &= set ? bb : ~bb;
            }
            const uint32_t leader = 31u - __clz(peers | 1u);
            uint32_t base = 0;
            if (valid && lane == leader) base = atomicAdd(&wh[d], (uint32_t)__popc(peers));
            pos[i] = __shfl_sync(0xffffffffu, base, (int)leader) + (uint32_t)__popc(peers & ltm);
        }
        gsync();  // every warp's counters are complete
        // exclusive scan over (digit, warp): thread gt owns digits gt*DPT .. gt*DPT+DPT-1 (the
        // counts are read again below rather than held in registers)
        uint32_t tot = 0;
        for (uint32_t j = 0; j < DPT; j++)
            for (uint32_t w = 0; w < G; w++) tot += s_whist[(gw0 + w) * 256 + gt * DPT + j];
        uint32_t inc = tot;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, d);
            if (lane >= (uint32_t)d) inc += y;
        }
        if (lane == 31) s_wsum[warp] = inc;
        gsync();
        uint32_t run = inc - tot;
        for (uint32_t w = 0; w < wg; w++) run += s_wsum[gw0 + w];
        for (uint32_t j = 0; j < DPT; j++)
            for (uint32_t w = 0; w < G; w++) {
                uint32_t* cw = &s_whist[(gw0 + w) * 256 + gt * DPT + j];
                const uint32_t c = *cw;
                *cw = run;
                run += c;
            }
        gsync();  // digit starts of every warp are in place
#pragma unroll
        for (int i = 0; i < ITEMS; i++) {
            const uint32_t r = (uint32_t)i * 32u + lane;
            if ((uint32_t)i >= IT || r >= wn) continue;
            const uint32_t q = pos[i] + wh[seg_digit<K, DESC>(k[i], shift)];
            sk[q] = k[i];
            vb[q] = va[wbase + r];
        }
        gsync();  // the pass's order is complete in sk / vb
        V* t = va; va = vb; vb = t;
        shift += 8u;
        if (p + 1 == plan.passes) {
            if (plan.shift == 0) break;
            // the last pass of the short form: the runs of tied keys
            if (sizeof(U) == 8 && plan.copies(Q0)) {
                const bool out =
                    __any_sync(0xffffffffu, seg_ties_inverted<K, DESC>(sk, wbase + lane, 32u, wbase + wn, len, plan.shift));
                if (lane == 0) wh[0] = out ? 1u : 0u;
                gsync();
                uint32_t any = 0;
                for (uint32_t w = 0; w < G; w++) any |= s_whist[(gw0 + w) * 256];
                gsync();  // the counters are free
                if (!any) break;
            }
            uint32_t fixed = __reduce_or_sync(
                0xffffffffu, seg_fix_runs<K, V, DESC>(sk, va, wbase + lane, 32u, wbase + wn, len, plan.shift));
            if (lane == 0) s_wsum[warp] = fixed;
            gsync();  // the runs are sorted
            fixed = 0;
            for (uint32_t w = 0; w < G; w++) fixed |= s_wsum[gw0 + w];
            if (!(fixed & (uint32_t)SEG_LONG)) break;
            bool inv = false;
            for (uint32_t r = lane; r < wn; r += 32u) inv |= seg_inverted<K, DESC>(sk, wbase + r);
            inv = __any_sync(0xffffffffu, inv);
            if (lane == 0) wh[0] = inv ? 1u : 0u;
            gsync();
            uint32_t any = 0;
            for (uint32_t w = 0; w < G; w++) any |= s_whist[(gw0 + w) * 256];
            gsync();  // the counters are free
            if (!any) break;
            plan = seg_full_plan(diff);
            shift = 0;
            p = ~0u;  // from the first pass again
        }
#pragma unroll
        for (int i = 0; i < ITEMS; i++) {
            const uint32_t r = (uint32_t)i * 32u + lane;
            if ((uint32_t)i < IT && r < wn) k[i] = sk[wbase + r];
        }
        // the next pass writes sk / vb only after its first group barrier, which every warp
        // reaches after this reload
    }
    // exclusive scan of the sorted values (in va; the sorted keys are in sk): warp totals, the
    // group's offsets, then each warp's rows with a running carry; keys, values and scan
    // written in element order
    V wsum = V();
#pragma unroll 1
    for (uint32_t r = lane; r < wn; r += 32u) wsum += va[wbase + r];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) wsum += shfl_xor_any(wsum, d);
    if (lane == 0) s_vpart[warp] = wsum;
    gsync();
    for (uint32_t w = 0; w < wg; w++) carry += s_vpart[gw0 + w];
#pragma unroll 1
    for (uint32_t r0 = 0; r0 < wn; r0 += 32u) {  // rows of the warp's chunk (warp-uniform)
        const uint32_t r = r0 + lane;
        const bool valid = r < wn;
        const V x = valid ? va[wbase + r] : V();
        V incl = x;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const V y = shfl_up_any(incl, d);
            if (lane >= (uint32_t)d) incl += y;
        }
        if (valid) {
            gk[wbase + r] = sk[wbase + r];
            gv[wbase + r] = x;
            if (gs) gs[wbase + r] = carry + incl - x;
        }
        carry += shfl_any(incl, 31);
    }
    gsync();  // s_vpart and the staging slices are free for the group's next segment
}

// One warp sorts (and scans) a segment of len <= 32 keys without digit counters: a bitonic
// network over (ordered code, original index) pairs, one per lane.  The index makes every
// pair distinct, so the network's result is the stable order (equal codes keep their input
// order); padding lanes carry the largest code and indices >= len, so they sort last.  Each
// lane then takes its key and value from the lane that held the element (shuffles only: the
// segment may be sorted in place).
template <class K, class V, bool DESC>
__device__ inline void seg_warp_bitonic(typename RadixKey<K>::B* gk, V* gv, V* gs, uint32_t len) {
    typedef typename RadixKey<K>::B KB;
    typedef typename RadixKey<K>::U U;
    const uint32_t lane = threadIdx.x & 31u;
    const bool valid = lane < len;
    const KB key = valid ? gk[lane] : KB(0);
    const V val = valid ? gv[lane] : V();
    U code = ~U(0);
    if (valid) {
        code = RadixKey<K>::ordered(key);
        if (DESC) code = ~code;
    }
    uint32_t idx = lane;
#pragma unroll
    for (uint32_t k = 2; k <= 32; k <<= 1) {
#pragma unroll
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            const U oc = __shfl_xor_sync(0xffffffffu, code, (int)j);
            const uint32_t oi = __shfl_xor_sync(0xffffffffu, idx, (int)j);
            const bool other_less = oc < code || (oc == code && oi < idx);
            // blocks of k alternate direction; the lower lane of a pair keeps the smaller
            // element in an ascending block and the larger one in a descending block
            const bool asc = (lane & k) == 0, lower = (lane & j) == 0;
            if ((asc == lower) == other_less) { code = oc; idx = oi; }
        }
    }
    const KB sk = shfl_any(key, (int)idx);
    const V sv = shfl_any(val, (int)idx);
    const V x = valid ? sv : V();
    V incl = x;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const V y = shfl_up_any(incl, d);
        if (lane >= (uint32_t)d) incl += y;
    }
    if (valid) {
        gk[lane] = sk;
        gv[lane] = sv;
        if (gs) gs[lane] = incl - x;
    }
}

template <class K, class V, int ITEMS>
constexpr size_t seg_sort_scan_smem() {
    return (size_t)256 * ITEMS * (2 * sizeof(V) + sizeof(typename RadixKey<K>::B)) + 8 * 256 * 4;
}

// One persistent launch over the whole batch.  keys/vals: the concatenated segments (sorted
// in place); scan: receives the exclusive scans; tk/tv: temp arrays of n elements (large
// segments only).
// resident CTAs per SM the batched kernel is compiled for (B200, 100k lognormal segments at 8
// items, u32 keys, all four passes per key: 2 CTAs (127 registers) 4.15 ms, 3 CTAs 3.53 ms, 4 CTAs (64 registers) 3.46 ms;
// 16 items need the shared memory of 3 CTAs; 8-byte keys keep 2 CTAs, which they fill without
// spilling)
#ifndef TRTC_SEG_MINB
#define TRTC_SEG_MINB(items, key_bytes) ((key_bytes) > 4 ? 2 : ((items) <= 8 ? 4 : 3))
#endif
// groups of two and four warps for the segments between one warp's share and a quarter of
// the CTA tile (0: those segments take the whole-CTA on-chip class)
#ifndef TRTC_SEG_GROUPS
#define TRTC_SEG_GROUPS 1
#endif
template <class K, class V, class OFF, bool DESC, int ITEMS, int MINB = TRTC_SEG_MINB(ITEMS, sizeof(K))>
__global__ void __launch_bounds__(256, MINB) seg_sort_scan_kernel(typename RadixKey<K>::B* __restrict__ keys,
                                                                V* __restrict__ vals, V* __restrict__ scan,
                                                                typename RadixKey<K>::B* __restrict__ tk,
                                                                V* __restrict__ tv, const OFF* __restrict__ off,
                                                                const uint32_t* __restrict__ queue,
                                                                unsigned long long nseg, SegCtrl* ctrl,
                                                                const SegItem* __restrict__ items,
                                                                uint32_t warp_small) {
    typedef typename RadixKey<K>::B KB;
    constexpr int TILE = 256 * ITEMS;
    constexpr int D = RadixKey<K>::DIGITS;
    extern __shared__ __align__(16) unsigned char seg_smem[];  // seg_sort_scan_smem<K, V, ITEMS>() bytes
    V* s_v = reinterpret_cast<V*>(seg_smem);
    V* s_o = s_v + TILE;
    KB* s_k = reinterpret_cast<KB*>(s_o + TILE);
    uint32_t* s_whist = reinterpret_cast<uint32_t*>(s_k + TILE);
    __shared__ uint32_t s_cnt[256], s_start[256], s_run[256];
    __shared__ uint32_t s_hist[D][256];
    __shared__ uint32_t s_wsum[8];
    __shared__ V s_part[8];
    __shared__ unsigned long long s_item;
    __shared__ unsigned long long s_batch, s_defer[8];
    __shared__ uint32_t s_bucket;
    static_assert(sizeof(typename RadixKey<K>::B) >= 4 && is_same<V, uint32_t>::value,
                  "keys of 4 or 8 bytes, uint32_t values");
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    constexpr uint32_t WSEG = 32u * ITEMS;  // segments up to this length are sorted by one warp

    // the arrays and length of queue entry `item`
    auto fetch = [&](unsigned long long item, KB*& gk, V*& gv, V*& gs, uint32_t& len, unsigned long long& base) {
        if (items) {  // list mode: segments in queue order, each with its own arrays
            const SegItem it = items[item];
            gk = reinterpret_cast<KB*>(it.k);
            gv = reinterpret_cast<V*>(it.v);
            gs = reinterpret_cast<V*>(it.out);
            len = (uint32_t)it.n;
            base = it.toff;
        } else {
            const uint32_t sid = queue[item];
            base = (unsigned long long)off[sid];
            len = (uint32_t)((unsigned long long)off[sid + 1] - base);
            gk = keys + base;
            gv = vals + base;
            gs = scan + base;
        }
    };

    // whole-CTA sort + scan of one segment (on chip up to TILE keys, else through global memory)
    auto block_segment = [&](KB* gk, V* gv, V* gs, uint32_t len, unsigned long long base) {
        typedef typename RadixKey<K>::U U;
        // OR over the CTA (in the digit counters, which every pass clears first)
        auto block_or = [&](U x) -> U {
            x = seg_warp_or(x);
            __syncthreads();
            if (lane == 0) {
                s_whist[2 * warp] = (uint32_t)x;
                s_whist[2 * warp + 1] = (uint32_t)((unsigned long long)x >> 32);
            }
            __syncthreads();
            for (int w = 0; w < 8; w++)
                x |= (U)(((unsigned long long)s_whist[2 * w + 1] << 32) | s_whist[2 * w]);
            __syncthreads();
            return x;
        };
        // eight samples spread over n >= 256 keys; two ties among uniform keys are 1 in 600
        auto sampled = [&](const KB* k, uint32_t n, uint32_t sh, bool dups) -> bool {
            const bool tie = seg_sample_ties(seg_code<K, DESC>(k[(n >> 8) * threadIdx.x]), true, sh, dups);
            return __syncthreads_count(tie && lane == 0) >= 2;
        };
        // finishes the runs of tied keys that a short form left; false: some run takes too long
        auto sorted = [&](const KB* k, uint32_t n) -> bool {
            bool inv = false;
            for (uint32_t e = threadIdx.x; e < n; e += 256) inv |= seg_inverted<K, DESC>(k, e);
            return !__syncthreads_or(inv);
        };
        auto fix_on_chip = [&](uint32_t n, const SegPlan& plan) -> bool {
            if (sizeof(U) == 8 && plan.copies(seg_min_passes<K>()) &&
                !__syncthreads_or(seg_ties_inverted<K, DESC>(s_k, threadIdx.x, 256u, n, n, plan.shift)))
                return true;
            const uint32_t fixed = seg_fix_runs<K, V, DESC>(s_k, s_v, threadIdx.x, 256u, n, n, plan.shift);
            if (!__syncthreads_or((int)(fixed & (uint32_t)SEG_LONG))) return true;
            return sorted(s_k, n);
        };
        // the same in global memory, where looking into every run of ties can cost more than the passes
        // saved: the first inverted tie of a run (walking back finds none before it) lists the run's
        // first key, in the digit counters, which every pass clears first
        auto fix_in_memory = [&](KB* k, V* v, uint32_t n, uint32_t shift) -> bool {
            if (threadIdx.x == 0) s_whist[0] = 0;
            __syncthreads();
            bool inv = false, far = false;
            for (uint32_t e = threadIdx.x; e + 1 < n; e += 256) {
                const U a = seg_code<K, DESC>(k[e]), b = seg_code<K, DESC>(k[e + 1]);
                if (((a ^ b) >> shift) != 0 || a <= b) continue;
                inv = true;
                uint32_t st = e;
                U next = a;
                bool lead = true;
                while (lead && st > 0) {
                    const U c = seg_code<K, DESC>(k[st - 1]);
                    if (((c ^ a) >> shift) != 0) break;
                    if (e - st >= (uint32_t)SEG_STEPS_FAR) far = true;
                    lead = c <= next && !far;
                    next = c;
                    st--;
                }
                if (!lead) continue;
                const uint32_t at = atomicAdd(&s_whist[0], 1u);
                if (at < 2047u) s_whist[1u + at] = st;
            }
            if (!__syncthreads_or(inv)) return true;
            const uint32_t runs = s_whist[0];
            if (__syncthreads_or(far) == 0 && runs <= 2047u) {
                uint32_t fixed = 0;
                for (uint32_t i = threadIdx.x; i < runs; i += 256)
                    fixed |= seg_fix_run<K, V, DESC, true>(k, v, s_whist[1u + i], n, shift);
                if (!__syncthreads_or((int)(fixed & (uint32_t)SEG_LONG))) return true;
            } else if (runs > 2047u) {
                uint32_t fixed = 0;
                fixed = seg_fix_runs<K, V, DESC>(k, v, threadIdx.x, 256u, n, n, shift);
                if (!__syncthreads_or((int)(fixed & (uint32_t)SEG_LONG))) return true;
            }
            return sorted(k, n);
        };
        // one stable pass by the digit at `shift` through global memory; s_run: the digits' starts
        auto scatter = [&](const KB* sk, const V* sv, KB* dk, V* dv, uint32_t shift) {
            for (uint32_t cb = 0; cb < len; cb += TILE) {
                const uint32_t cn = min((uint32_t)TILE, len - cb);
                const int IT = (int)((cn + 255u) / 256u);
                const uint32_t wbase = warp * 32u * (uint32_t)IT;
                KB k[ITEMS];
                V v[ITEMS];
                uint32_t pos[ITEMS];
#pragma unroll
                for (int i = 0; i < ITEMS; i++) {
                    const uint32_t e = wbase + (uint32_t)i * 32u + lane;
                    if (i < IT && e < cn) { k[i] = sk[cb + e]; v[i] = sv[cb + e]; }
                    else { k[i] = KB(0); v[i] = V(); }
                }
                seg_rank_tile<K, DESC, ITEMS>(k, pos, IT, cn, shift, s_whist, s_cnt, s_start, s_wsum);
#pragma unroll
                for (int i = 0; i < ITEMS; i++) {
                    const uint32_t e = wbase + (uint32_t)i * 32u + lane;
                    if (i < IT && e < cn) { s_k[pos[i]] = k[i]; s_v[pos[i]] = v[i]; }
                }
                __syncthreads();
                for (uint32_t e = threadIdx.x; e < cn; e += 256) {
                    const KB key = s_k[e];
                    const uint32_t d = seg_digit<K, DESC>(key, shift);
                    const uint32_t dst = s_run[d] + (e - s_start[d]);
                    dk[dst] = key;
                    dv[dst] = s_v[e];
                }
                __syncthreads();
                s_run[threadIdx.x] += s_cnt[threadIdx.x];
                __syncthreads();
            }
        };
        const KB* ck = gk;  // what the on-chip part reads: the segment, or its buckets in tk / tv
        const V* cv = gv;
        const bool split = len > (uint32_t)TILE;
        if (split) {
            // ---------------- large segment
            KB* dk = tk + base;
            V* dv = tv + base;
            const U ref = seg_code<K, DESC>(gk[0]);
            // from two CTA tiles up, four of floats (16 keys a thread: 8192 and 16,384 keys; 2^24 u32 keys in
            // segments of 40,000: 829 us by LSD passes, 598 this way, one segment of 100,000 951 and 667; of
            // 9000 717 and 678; f32 of 14,000 824 and 858; i64 of 9000 1757 and 1102).  4-byte keys of 2.5 to
            // 3 tiles, where LSD passes run over full tiles and there would be twice the buckets, half as
            // full: u32 of 12,000 655 and 719, one of them 133 and 149, one of 10,291 123 and 144.
            // one pass by the top bits of those that vary puts the keys into buckets of 5/8 of a
            // warp's share on average (up to 256 of them); each is then sorted on chip.  Which bits
            // vary is read off a sample of 256 keys and checked by the pass that counts them all.
            const KB sample = gk[(len >> 8) * threadIdx.x];
            U diff = block_or(seg_code<K, DESC>(sample) ^ ref);
            const uint32_t bits = diff ? 64u - (uint32_t)__clzll((long long)(unsigned long long)diff) : 1u;
            const uint32_t nb = min(8u, 32u - (uint32_t)__clz((len - 1u) / (WSEG * 5u / 8u)));
            const uint32_t top = bits > nb ? bits - nb : 0u;
            s_hist[0][threadIdx.x] = 0;
            s_hist[1][threadIdx.x] = 0;
            __syncthreads();
            atomicAdd(&s_hist[0][seg_digit<K, DESC>(sample, top)], 1u);
            __syncthreads();
            // (clustered keys, the exponents of floats, fill a bucket: seen in the sample already.)  With
            // many copies a bucket that is too large is certain sooner, and 4-byte keys take the LSD
            // passes (u32 ids of a Zipf popularity in segments of 10,000: 702 us, in buckets 1098)
            const uint32_t seen = s_hist[0][threadIdx.x];
            const bool copies = __syncthreads_count(seg_sample_ties(seg_code<K, DESC>(sample), true, 0u, true) && lane == 0) >= 2;
            const bool few = seg_min_passes<K>() == 3u ? len <= 4u * (uint32_t)TILE
                                                       : len <= 2u * (uint32_t)TILE ||
                                                             (sizeof(U) == 4 && len > 5u * (uint32_t)TILE / 2u && len <= 3u * (uint32_t)TILE);
            bool one = __syncthreads_or(few || (sizeof(U) == 4 && copies) ||
                                        (seen >= 16u && (unsigned long long)seen * (len >> 8) > (copies ? 1ull : 2ull) * TILE));
            if (!one) {
                s_hist[0][threadIdx.x] = 0;
                __syncthreads();
                U all = 0;
                for (uint32_t e = threadIdx.x; e < len; e += 1024) {
                    KB k[4];
                    V v[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const uint32_t x = min(e + 256u * j, len - 1u);
                        k[j] = gk[x];
                        v[j] = gv[x];
                    }
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        all |= seg_code<K, DESC>(k[j]) ^ ref;
                        if (e + 256u * j >= len) continue;
                        const uint32_t d = seg_digit<K, DESC>(k[j], top);
                        atomicAdd(&s_hist[0][d], 1u);
                        atomicAdd(&s_hist[1][d], (uint32_t)v[j]);
                    }
                }
                __syncthreads();
                const uint32_t c = s_hist[0][threadIdx.x], sum = s_hist[1][threadIdx.x];
                one = __syncthreads_or(c > (uint32_t)TILE || (all >> top) > U(0xFF));
                if (!one) {
                    const uint32_t st = block_excl_scan_256<256>(c, s_wsum);
                    __syncthreads();
                    s_hist[2][threadIdx.x] = block_excl_scan_256<256>(sum, s_wsum);  // the scan's value at the bucket
                    s_hist[1][threadIdx.x] = st;
                    s_run[threadIdx.x] = st;
                    __syncthreads();
                    scatter(gk, gv, dk, dv, top);
                    if (threadIdx.x == 0) s_bucket = 0;
                    __syncthreads();
                    // buckets of up to a warp's share: one warp each
                    while (true) {
                        uint32_t b = 0;
                        if (lane == 0) b = atomicAdd(&s_bucket, 1u);
                        b = __shfl_sync(0xffffffffu, b, 0);
                        if (b >= 256u) break;
                        const uint32_t n = s_hist[0][b], o = s_hist[1][b];
                        if (n == 0 || n > WSEG) continue;
                        seg_warp_sort_scan<K, V, DESC, ITEMS>(dk + o, dv + o, gk + o, gv + o, gs ? gs + o : nullptr, n,
                                                              (V)s_hist[2][b], s_k + warp * WSEG, s_v + warp * WSEG,
                                                              s_whist + warp * 256);
                    }
                    __syncthreads();
                    // up to two and four shares: groups of two and four warps
                    for (uint32_t G = 2; G <= 4; G *= 2) {
                        const uint32_t grp = warp / G;
                        for (uint32_t b = grp; b < 256u; b += 8u / G) {
                            const uint32_t n = s_hist[0][b], o = s_hist[1][b];
                            if (n <= G / 2 * WSEG || n > G * WSEG) continue;
                            seg_group_sort_scan<K, V, DESC, ITEMS>(
                                dk + o, dv + o, gk + o, gv + o, gs ? gs + o : nullptr, n, (V)s_hist[2][b],
                                s_k + grp * G * WSEG, s_v + grp * G * WSEG, s_o + grp * G * WSEG, s_whist, s_wsum,
                                s_part, G, 1u + grp);
                        }
                        __syncthreads();
                    }
                    ck = dk;
                    cv = dv;
                }
            }
            if (one) {
                // CTA-level LSD passes through global memory
                KB* sk = gk;
                V* sv = gv;
                SegPlan plan;
                if constexpr (sizeof(U) == 8) {
                    diff = 0;
#pragma unroll 4
                    for (uint32_t e = threadIdx.x; e < len; e += 256) diff |= seg_code<K, DESC>(gk[e]) ^ ref;
                    diff = block_or(diff);
                    plan = seg_plan(diff, len, 3u, 1u << 16, [&](uint32_t sh, bool dups) { return sampled(gk, len, sh, dups); });
                } else {  // (finding the varying bits, three passes and the ties cost as much as four passes)
                    diff = ~U(0);
                    plan = seg_full_plan(diff);
                }
                while (true) {
                    for (uint32_t i = threadIdx.x; i < plan.passes * 256u; i += 256u) (&s_hist[0][0])[i] = 0;
                    __syncthreads();
                    for (uint32_t e = threadIdx.x; e < len; e += 256) {
                        const U u = seg_code<K, DESC>(sk[e]) >> plan.shift;
#pragma unroll
                        for (int p = 0; p < D; p++) {
                            if ((uint32_t)p >= plan.passes) break;
                            const uint32_t w = (p < 4) ? (uint32_t)u : (uint32_t)((unsigned long long)u >> 32);
                            atomicAdd(&s_hist[p][__byte_perm(w, 0u, 0x4440u | (uint32_t)(p & 3))], 1u);
                        }
                    }
                    __syncthreads();
                    for (uint32_t p = 0; p < plan.passes; p++) {
                        const uint32_t shift = plan.shift + 8u * p;
                        {
                            const uint32_t c = s_hist[p][threadIdx.x];
                            s_run[threadIdx.x] = block_excl_scan_256<256>(c, s_wsum);
                        }
                        __syncthreads();
                        scatter(sk, sv, dk, dv, shift);
                        KB* t1 = sk; sk = dk; dk = t1;
                        V* t2 = sv; sv = dv; dv = t2;
                    }
                    if (plan.shift == 0 || fix_in_memory(sk, sv, len, plan.shift)) break;
                    plan = seg_full_plan(diff);
                }
                // the sorted segment is in sk/sv (the caller's arrays after an even number of passes);
                // chunked exclusive scan with a running carry, writing keys and values back if needed
                V carry = V();
                for (uint32_t cb = 0; cb < len; cb += TILE) {
                    const uint32_t cn = min((uint32_t)TILE, len - cb);
                    for (uint32_t e = threadIdx.x; e < cn; e += 256) {
                        s_v[e] = sv[cb + e];
                        if (sk != gk) { gk[cb + e] = sk[cb + e]; gv[cb + e] = s_v[e]; }
                    }
                    __syncthreads();
                    if (gs) {
                        carry = seg_block_excl_scan<V, ITEMS>(s_v, s_o, cn, carry, s_part);
                        for (uint32_t e = threadIdx.x; e < cn; e += 256) gs[cb + e] = s_o[e];
                    }
                    __syncthreads();
                }
                return;
            }
        }

        // ---------------- on-chip sort: the segment, or the buckets above four shares
        for (uint32_t b = 0; b < (split ? 256u : 1u); b++) {
            const uint32_t n = split ? s_hist[0][b] : len, st = split ? s_hist[1][b] : 0u;
            if (split && n <= 4u * WSEG) continue;
            const V first = split ? (V)s_hist[2][b] : V();
            const KB* ik = ck + st;
            const V* iv = cv + st;
            const int IT = (int)((n + 255u) / 256u);
            const uint32_t wbase = warp * 32u * (uint32_t)IT;
            KB k[ITEMS];
            V v[ITEMS];
            uint32_t pos[ITEMS];
#pragma unroll
            for (int i = 0; i < ITEMS; i++) {
                const uint32_t e = wbase + (uint32_t)i * 32u + lane;
                if (i < IT && e < n) { k[i] = ik[e]; v[i] = iv[e]; }
                else { k[i] = KB(0); v[i] = V(); }
            }
            const U ref = seg_code<K, DESC>(ik[0]);
            U diff = 0;
#pragma unroll
            for (int i = 0; i < ITEMS; i++)
                if (i < IT && wbase + (uint32_t)i * 32u + lane < n) diff |= seg_code<K, DESC>(k[i]) ^ ref;
            diff = block_or(diff);
            SegPlan plan = seg_plan(diff, n, seg_min_passes<K>(), seg_dups3<K>(),
                                    [&](uint32_t sh, bool dups) { return sampled(ik, n, sh, dups); });
            uint32_t shift = plan.shift;
            for (uint32_t p = 0; p < plan.passes; p++) {
                seg_rank_tile<K, DESC, ITEMS>(k, pos, IT, n, shift, s_whist, s_cnt, s_start, s_wsum);
#pragma unroll
                for (int i = 0; i < ITEMS; i++) {
                    const uint32_t e = wbase + (uint32_t)i * 32u + lane;
                    if (i < IT && e < n) { s_k[pos[i]] = k[i]; s_v[pos[i]] = v[i]; }
                }
                __syncthreads();
                shift += 8u;
                if (p + 1 == plan.passes) {
                    if (plan.shift == 0 || fix_on_chip(n, plan)) break;
                    plan = seg_full_plan(diff);
                    shift = 0;
                    p = ~0u;  // from the first pass again
                }
#pragma unroll
                for (int i = 0; i < ITEMS; i++) {
                    const uint32_t e = wbase + (uint32_t)i * 32u + lane;
                    if (i < IT && e < n) { k[i] = s_k[e]; v[i] = s_v[e]; }
                }
                __syncthreads();
            }
            // s_k / s_v hold the sorted segment; exclusive scan of the values into s_o
            if (gs) seg_block_excl_scan<V, ITEMS>(s_v, s_o, n, first, s_part);
            for (uint32_t e = threadIdx.x; e < n; e += 256) {
                gk[st + e] = s_k[e];
                gv[st + e] = s_v[e];
                if (gs) gs[st + e] = s_o[e];
            }
        }
    };

    while (true) {
        __syncthreads();
        if (threadIdx.x == 0) s_item = atomicAdd(&ctrl->next, 1ull);
        __syncthreads();
        const unsigned long long item = s_item;
        if (item >= nseg) return;
        KB* gk;
        V* gv;
        V* gs;
        uint32_t len;
        unsigned long long base;
        fetch(item, gk, gv, gs, len, base);
        if (len == 0) continue;
        // a segment of the CTA classes is sorted by the whole CTA below (one copy of that code).
        // A small one: the queue lists the classes from the largest down, so the entries
        // after it are no longer than its class.  The CTA splits into groups of G warps (one
        // warp up to WSEG keys, two up to 2 WSEG, four up to 4 WSEG), takes one more entry per
        // further group, and every group sorts one; an entry longer than its group's share
        // (list mode keeps the caller's order) is deferred to the whole CTA afterwards
        const uint32_t G = !TRTC_SEG_GROUPS ? 1u : len > 2u * WSEG ? 4u : (len > WSEG ? 2u : 1u);  // CTA-uniform
        unsigned long long defer = warp == 0 ? item : ~0ull;
        if (len <= (TRTC_SEG_GROUPS ? 4u : 1u) * WSEG) {  // CTA-uniform
            if (threadIdx.x == 0) s_batch = atomicAdd(&ctrl->next, (unsigned long long)(8u / G - 1u));
            __syncthreads();
            const uint32_t grp = warp / G;
            const unsigned long long mine = grp == 0 ? item : s_batch + grp - 1;
            defer = ~0ull;
            if (mine < nseg) {
                KB* wk;
                V* wv;
                V* ws;
                uint32_t wl;
                unsigned long long wb;
                fetch(mine, wk, wv, ws, wl, wb);
                if (wl > G * WSEG) defer = mine;
                else if (wl > 0 && G == 1 && wl <= warp_small) seg_warp_bitonic<K, V, DESC>(wk, wv, ws, wl);
                else if (wl > 0 && G == 1)
                    seg_warp_sort_scan<K, V, DESC, ITEMS>(wk, wv, wk, wv, ws, wl, V(), s_k + warp * WSEG,
                                                          s_v + warp * WSEG, s_whist + warp * 256);
                else if (wl > 0)
                    seg_group_sort_scan<K, V, DESC, ITEMS>(wk, wv, wk, wv, ws, wl, V(), s_k + grp * G * WSEG,
                                                           s_v + grp * G * WSEG, s_o + grp * G * WSEG, s_whist, s_wsum,
                                                           s_part, G, 1u + grp);
            }
        }
        if (lane == 0) s_defer[warp] = (warp % G == 0) ? defer : ~0ull;
        __syncthreads();
        for (int w = 0; w < 8; w++) {
            const unsigned long long d = s_defer[w];
            if (d == ~0ull) continue;
            fetch(d, gk, gv, gs, len, base);
            block_segment(gk, gv, gs, len, base);
            __syncthreads();
        }
    }
}

// ------------------------------------------------------------------ NaN rotation (float keys)
// The reference sorts a float vector by (code(x) - code(m)) mod 2^w, m the element that its
// Min_Element tree selects (extrema.cpp:5-13 over internal/general_reduce.cpp:55-95).  With a
// NaN in a left slot the tree can select a non-minimum, and the sorted order is the code order
// rotated so that the keys ordered at or above m come first.  A segment sorted on its own gets
// the same rotation here: seg_rot_kernel (before the sort) replays the tree on every segment
// that holds a NaN and counts its keys ordered strictly below the selected one;
// seg_rotate_kernel (after the sort) rotates those segments by that count and redoes their
// exclusive scans.  Segments without a NaN are only read once, for the NaN test.
template <class K> struct SegMinSlot {
    K v;
    unsigned long long i;
};

// tree slots of a segment starting at element `base` (index `sid`): the rounds need at most
// ceil(L/256) + ceil(L/2^16) + ceil(L/2^24) + 1 slots, which fit between base/128 + 4*sid and
// the next segment's start; the whole area holds n/128 + 4*nseg + 4 slots
TRTC_FORCEINLINE unsigned long long seg_tree_base(unsigned long long base, unsigned long long sid) {
    return base / 128ull + 4ull * sid;
}
inline unsigned long long seg_tree_slots(unsigned long long n, unsigned long long nseg) {
    return n / 128ull + 4ull * nseg + 4ull;
}

template <class K, class OFF>
__global__ void __launch_bounds__(256) seg_rot_kernel(const typename RadixKey<K>::B* __restrict__ keys,
                                                      const OFF* __restrict__ off,
                                                      const SegItem* __restrict__ items, unsigned long long nseg,
                                                      SegMinSlot<K>* tree, uint32_t* __restrict__ rot) {
    typedef RadixKey<K> RK;
    typedef typename RK::B KB;
    __shared__ unsigned long long s_c[8];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    for (unsigned long long sid = blockIdx.x; sid < nseg; sid += gridDim.x) {
        const KB* gk;
        uint32_t len;
        unsigned long long base;
        if (items) {
            const SegItem it = items[sid];
            gk = reinterpret_cast<const KB*>(it.k);
            len = (uint32_t)it.n;
            base = it.toff;
        } else {
            base = (unsigned long long)off[sid];
            len = (uint32_t)((unsigned long long)off[sid + 1] - base);
            gk = keys + base;
        }
        bool nan = false;
        for (uint32_t e = threadIdx.x; e < len; e += 256) nan |= RK::is_nan(gk[e]);
        if (!__syncthreads_or(nan)) {
            if (threadIdx.x == 0) rot[sid] = 0;
            continue;
        }
        // round 1 over 256-blocks of the keys, then rounds over the block results (slots in
        // global memory, written and read by this CTA only, ordered by its barriers)
        SegMinSlot<K>* src = tree + seg_tree_base(base, sid);
        uint32_t m = (len + 255u) / 256u;
        for (uint32_t b = warp; b < m; b += 8) {
            const uint32_t L = min(256u, len - b * 256u);
            K rv;
            unsigned long long ri;
            min_tree_warp256<K>(
                [&](uint32_t t, K& v, unsigned long long& i) { v = RK::value(gk[b * 256u + t]); i = b * 256u + t; },
                L, rv, ri);
            if (lane == 0) { src[b].v = rv; src[b].i = ri; }
        }
        __syncthreads();
        while (m > 1) {
            SegMinSlot<K>* dst = src + m;
            const uint32_t nb = (m + 255u) / 256u;
            for (uint32_t b = warp; b < nb; b += 8) {
                const uint32_t L = min(256u, m - b * 256u);
                K rv;
                unsigned long long ri;
                min_tree_warp256<K>(
                    [&](uint32_t t, K& v, unsigned long long& i) { v = src[b * 256u + t].v; i = src[b * 256u + t].i; },
                    L, rv, ri);
                if (lane == 0) { dst[b].v = rv; dst[b].i = ri; }
            }
            __syncthreads();
            src = dst;
            m = nb;
        }
        const typename RK::U tm = RK::ordered(gk[src[0].i]);
        unsigned long long c = 0;
        for (uint32_t e = threadIdx.x; e < len; e += 256) c += RK::ordered(gk[e]) < tm ? 1ull : 0ull;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) c += __shfl_down_sync(0xffffffffu, c, d);
        if (lane == 0) s_c[warp] = c;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned long long t = 0;
            for (int w = 0; w < 8; w++) t += s_c[w];
            rot[sid] = (uint32_t)t;
        }
        __syncthreads();
    }
}

template <class K, class V, class OFF, bool DESC>
__global__ void __launch_bounds__(256) seg_rotate_kernel(typename RadixKey<K>::B* __restrict__ keys,
                                                         V* __restrict__ vals, V* __restrict__ scan,
                                                         typename RadixKey<K>::B* __restrict__ tk,
                                                         V* __restrict__ tv, const OFF* __restrict__ off,
                                                         const SegItem* __restrict__ items, unsigned long long nseg,
                                                         const uint32_t* __restrict__ rot) {
    typedef typename RadixKey<K>::B KB;
    constexpr int CH = 1024;
    __shared__ V s_v[CH], s_o[CH], s_part[8];
    for (unsigned long long sid = blockIdx.x; sid < nseg; sid += gridDim.x) {
        const uint32_t r = rot[sid];
        if (r == 0) continue;
        KB* gk;
        V *gv, *gs;
        uint32_t len;
        unsigned long long base;
        if (items) {
            const SegItem it = items[sid];
            gk = reinterpret_cast<KB*>(it.k);
            gv = reinterpret_cast<V*>(it.v);
            gs = reinterpret_cast<V*>(it.out);
            len = (uint32_t)it.n;
            base = it.toff;
        } else {
            base = (unsigned long long)off[sid];
            len = (uint32_t)((unsigned long long)off[sid + 1] - base);
            gk = keys + base;
            gv = vals + base;
            gs = scan + base;
        }
        for (uint32_t e = threadIdx.x; e < len; e += 256) { tk[base + e] = gk[e]; tv[base + e] = gv[e]; }
        __syncthreads();
        // ascending: sorted position p moves to p - r (mod len); descending: to p + r
        for (uint32_t e = threadIdx.x; e < len; e += 256) {
            uint32_t d = DESC ? e + r : e + (len - r);
            if (d >= len) d -= len;
            gk[d] = tk[base + e];
            gv[d] = tv[base + e];
        }
        __syncthreads();
        if (gs) {
            V carry = V();
            for (uint32_t cb = 0; cb < len; cb += CH) {
                const uint32_t cn = min((uint32_t)CH, len - cb);
                for (uint32_t e = threadIdx.x; e < cn; e += 256) s_v[e] = gv[cb + e];
                __syncthreads();
                carry = seg_block_excl_scan<V, CH / 256>(s_v, s_o, cn, carry, s_part);
                for (uint32_t e = threadIdx.x; e < cn; e += 256) gs[cb + e] = s_o[e];
                __syncthreads();
            }
        }
    }
}

// Exclusive Plus scans of many segments (list mode): a persistent CTA takes one segment at
// a time and scans it in chunks of 256 * ITEMS with a running carry.
template <class T, int ITEMS>
__global__ void __launch_bounds__(256) seg_scan_list_kernel(const SegItem* __restrict__ items, unsigned long long nseg,
                                                            SegCtrl* ctrl) {
    constexpr int TILE = 256 * ITEMS;
    __shared__ __align__(16) T s_v[TILE];
    __shared__ __align__(16) T s_o[TILE];
    __shared__ T s_part[8];
    __shared__ unsigned long long s_item;
    while (true) {
        __syncthreads();
        if (threadIdx.x == 0) s_item = atomicAdd(&ctrl->next, 1ull);
        __syncthreads();
        const unsigned long long item = s_item;
        if (item >= nseg) return;
        const SegItem it = items[item];
        const T* in = reinterpret_cast<const T*>(it.k);
        T* out = reinterpret_cast<T*>(it.out);
        T carry = T();
        for (unsigned long long cb = 0; cb < it.n; cb += TILE) {
            const uint32_t cn = (uint32_t)min((unsigned long long)TILE, it.n - cb);
            for (uint32_t e = threadIdx.x; e < cn; e += 256) s_v[e] = in[cb + e];
            __syncthreads();
            carry = seg_block_excl_scan<T, ITEMS>(s_v, s_o, cn, carry, s_part);
            for (uint32_t e = threadIdx.x; e < cn; e += 256) out[cb + e] = s_o[e];
            __syncthreads();
        }
    }
}

// Plus reductions of many segments (list mode); the result of segment i goes to
// *(T*)items[i].out.
template <class T>
__global__ void __launch_bounds__(256) seg_reduce_list_kernel(const SegItem* __restrict__ items, unsigned long long nseg,
                                                              SegCtrl* ctrl) {
    __shared__ T s_w[8];
    __shared__ unsigned long long s_item;
    while (true) {
        __syncthreads();
        if (threadIdx.x == 0) s_item = atomicAdd(&ctrl->next, 1ull);
        __syncthreads();
        const unsigned long long item = s_item;
        if (item >= nseg) return;
        const SegItem it = items[item];
        const T* in = reinterpret_cast<const T*>(it.k);
        T a = T();
        for (unsigned long long e = threadIdx.x; e < it.n; e += 256) a += in[e];
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) a += shfl_down_any(a, d);
        if ((threadIdx.x & 31u) == 0) s_w[threadIdx.x >> 5] = a;
        __syncthreads();
        if (threadIdx.x == 0) {
            T t = s_w[0];
            for (int w = 1; w < 8; w++) t += s_w[w];
            *reinterpret_cast<T*>(it.out) = t;
        }
    }
}

}  // namespace trtc
