// trtc_merge.cuh -- stable comparison sort for user comparators, and generic view copies.
//
// The reference sorts with a user Functor comparator (or non-radix key types) through a
// merge sort (internal/merge_sort.cpp:7-280): 512-element block sorts in shared memory,
// then pairwise merges of sorted runs where every element finds its output position by a
// binary search in the partner run.  Here both steps split work by merge-path diagonals
// (Green, McColl, Bader 2012): a worker that owns outputs [d, d + k) of a merge finds how many
// of the d outputs before it come from the left run by one binary search along diagonal d,
// then merges k outputs serially.  Ties take the left run first, which keeps the sort stable.
//   * block sort: a thread sorts ITEMS consecutive elements in registers (odd-even
//     transposition, swapping only a strictly smaller right neighbour), then the CTA merges
//     runs of ITEMS, 2*ITEMS, ... in shared memory, each thread ITEMS outputs per round;
//   * merge level: a CTA owns BLOCK*ITEMS consecutive outputs, two warps find its two
//     diagonals by 32-way searches, the CTA loads exactly the keys it merges (coalesced, the
//     whole tile once), every thread merges ITEMS outputs and records where each came from,
//     and the tile's keys and values are written coalesced in output order.
// A level moves every key and value once (16 B per 8-byte pair); per element it costs one
// comparison and a search of log2(tile) / ITEMS comparisons, where a search per element costs
// log2(run) comparisons on dependent global loads.  Measured times and what bounds them stand
// at merge_sort_impl.
// An inconsistent comparator (NaN under <) leaves an unspecified order, as before, but every
// access stays inside its run: the diagonals of a tile are clamped to what the runs hold.
#pragma once
#include "trtc_prelude.cuh"
#include "trtc_builtins.cuh"

namespace trtc {

// Shared-memory slot of tile element i.  In the block sort threads start their merges about
// ITEMS / 2 elements apart, which would put a warp on a few banks: PAD adds a slot every 32.
template <bool PAD> TRTC_FORCEINLINE uint32_t merge_slot(uint32_t i) { return PAD ? i + (i >> 5) : i; }

// ITEMS consecutive 2-byte source indices of a thread into shared memory, in 16-byte stores
// where they fill whole ones
template <int ITEMS> TRTC_FORCEINLINE void merge_store_from(unsigned short* s, const unsigned short (&v)[ITEMS]) {
    if constexpr (ITEMS % 8 == 0) {
        union U { uint4 q[ITEMS / 8]; unsigned short t[ITEMS]; TRTC_FORCEINLINE U() {} } u;
#pragma unroll
        for (int i = 0; i < ITEMS; i++) u.t[i] = v[i];
#pragma unroll
        for (int i = 0; i < ITEMS / 8; i++) reinterpret_cast<uint4*>(s)[i] = u.q[i];
    } else {
#pragma unroll
        for (int i = 0; i < ITEMS; i++) s[i] = v[i];
    }
}

// Serial merge of ITEMS outputs of the sorted tile ranges [a, a_end) and [b, b_end): the tile
// index each output came from.  The next key of a range is read unconditionally, so s_k has one
// slot more than the tile; outputs past the ranges' end are unspecified.  A warp whose threads
// all have ITEMS elements left in both ranges needs no end test (FULL: all 32 lanes call this;
// one choice for the warp, since lanes on both paths would run both).
template <class K, class Comp, int ITEMS, bool PAD, bool FULL>
TRTC_FORCEINLINE void merge_serial(const K* s_k, uint32_t a, uint32_t a_end, uint32_t b, uint32_t b_end, Comp& comp,
                                   unsigned short (&from)[ITEMS]) {
    K ka = s_k[merge_slot<PAD>(a)], kb = s_k[merge_slot<PAD>(b)];
    bool inner = false;
    if constexpr (FULL) inner = __all_sync(0xffffffffu, a + ITEMS <= a_end && b + ITEMS <= b_end);
    if (inner) {
#pragma unroll
        for (int i = 0; i < ITEMS; i++) {
            const bool tb = (bool)comp(kb, ka);
            from[i] = (unsigned short)(tb ? b : a);
            const uint32_t x = (tb ? b : a) + 1u;
            const K kx = s_k[merge_slot<PAD>(x)];
            if (tb) { b = x; kb = kx; } else { a = x; ka = kx; }
        }
    } else {
#pragma unroll
        for (int i = 0; i < ITEMS; i++) {
            const bool tb = b < b_end && (a >= a_end || (bool)comp(kb, ka));
            from[i] = (unsigned short)(tb ? b : a);
            uint32_t x = (tb ? b : a) + 1u;
            x = x < b_end ? x : b_end;  // stays inside the tile once both ranges are used up
            const K kx = s_k[merge_slot<PAD>(x)];
            if (tb) { b = x; kb = kx; } else { a = x; ka = kx; }
        }
    }
}

// how many of the first d outputs of merging tile ranges [a0, a0 + na) and [b0, b0 + nb) come
// from the left one
template <class K, class Comp, bool PAD>
TRTC_FORCEINLINE uint32_t merge_path_tile(const K* s_k, uint32_t a0, uint32_t na, uint32_t b0, uint32_t nb, uint32_t d,
                                          Comp& comp) {
    uint32_t lo = d > nb ? d - nb : 0u, hi = d < na ? d : na;
    while (lo < hi) {
        const uint32_t m = (lo + hi) >> 1;
        const K kb = s_k[merge_slot<PAD>(b0 + d - 1 - m)];
        const K ka = s_k[merge_slot<PAD>(a0 + m)];
        if ((bool)comp(kb, ka)) hi = m; else lo = m + 1;
    }
    return lo;
}

// One element global -> shared, asynchronously (no register held until it arrives) for the
// sizes cp.async has.
template <class T> TRTC_FORCEINLINE void merge_copy_async(T* s, const T* g) {
    if constexpr (sizeof(T) == 4 || sizeof(T) == 8 || (sizeof(T) == 16 && alignof(T) == 16)) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(s)), "l"(g),
                     "n"((int)sizeof(T)) : "memory");
    } else {
        *s = *g;
    }
}
TRTC_FORCEINLINE void merge_copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <bool B> struct MergeBool { static constexpr bool value = B; };

template <class KV, class VV, class OKV, class OVV, class Comp, bool HAS_VALS, int BLOCK, int ITEMS>
__global__ void __launch_bounds__(BLOCK) merge_block_sort_kernel(KV keys, VV vals, OKV out_k, OVV out_v, Comp comp,
                                                                 size_t n) {
    typedef typename remove_cvref<typename KV::value_t>::type K;
    constexpr uint32_t T = BLOCK * ITEMS;
    constexpr bool PAD = sizeof(K) <= 8;
    __shared__ __align__(16) K s_k[T + 1 + (PAD ? T / 32 : 0)];
    __shared__ __align__(16) unsigned short s_from[HAS_VALS ? T : 8];
    const size_t base = (size_t)blockIdx.x * T;
    const uint32_t cnt = (uint32_t)((n - base) < (size_t)T ? (n - base) : (size_t)T);
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
        const uint32_t p = (uint32_t)i * BLOCK + threadIdx.x;
        if (p < cnt) s_k[merge_slot<PAD>(p)] = keys[base + p];
    }
    __syncthreads();
    const uint32_t t0 = threadIdx.x * ITEMS;
    const uint32_t mine = cnt <= t0 ? 0u : (cnt - t0 < (uint32_t)ITEMS ? cnt - t0 : (uint32_t)ITEMS);
    K k[ITEMS];
    unsigned short from[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
        k[i] = s_k[merge_slot<PAD>(t0 + i)];
        from[i] = (unsigned short)(t0 + i);
    }
    // slots past cnt hold unspecified values that no merge reads as part of a range
    auto store_tile = [&]() {
#pragma unroll
        for (int i = 0; i < ITEMS; i++) s_k[merge_slot<PAD>(t0 + i)] = k[i];
        if constexpr (HAS_VALS) merge_store_from<ITEMS>(s_from + t0, from);
    };
    auto sort_tile = [&](auto full_c) {
        constexpr bool FULL = decltype(full_c)::value;
#pragma unroll
        for (int r = 0; r < ITEMS; r++) {
#pragma unroll
            for (int i = r & 1; i + 1 < ITEMS; i += 2) {
                if ((FULL || i + 1 < (int)mine) && (bool)comp(k[i + 1], k[i])) {
                    const K x = k[i]; k[i] = k[i + 1]; k[i + 1] = x;
                    const unsigned short y = from[i]; from[i] = from[i + 1]; from[i + 1] = y;
                }
            }
        }
        __syncthreads();
        store_tile();
        for (uint32_t w = ITEMS; w < T && (FULL || w < cnt); w *= 2) {
            __syncthreads();
            const uint32_t a0 = t0 & ~(2u * w - 1u);  // 2w is a power of two
            uint32_t mid = a0 + w, end = a0 + 2u * w;
            if (!FULL) { mid = mid < cnt ? mid : cnt; end = end < cnt ? end : cnt; }
            if (FULL || mine > 0) {
                unsigned short src[ITEMS];
                const uint32_t d = t0 - a0;
                const uint32_t pa = merge_path_tile<K, Comp, PAD>(s_k, a0, mid - a0, mid, end - mid, d, comp);
                merge_serial<K, Comp, ITEMS, PAD, FULL>(s_k, a0 + pa, mid, mid + d - pa, end, comp, src);
#pragma unroll
                for (int i = 0; i < ITEMS; i++) {
                    const uint32_t f = src[i];
                    k[i] = s_k[merge_slot<PAD>(f)];
                    if constexpr (HAS_VALS) from[i] = s_from[FULL || f < T ? f : 0u];
                }
            }
            __syncthreads();
            if (FULL || mine > 0) store_tile();
        }
        __syncthreads();
    };
    if (cnt == T) sort_tile(MergeBool<true>()); else sort_tile(MergeBool<false>());
    // a tile written over its own input (one tile in all) reads all its values first
    typedef typename remove_cvref<typename OKV::value_t>::type OK;
    if constexpr (HAS_VALS) {
        typedef typename remove_cvref<typename OVV::value_t>::type OV;
        OV v[ITEMS];
#pragma unroll
        for (int i = 0; i < ITEMS; i++) {
            const uint32_t p = (uint32_t)i * BLOCK + threadIdx.x;
            if (p < cnt) v[i] = (OV)vals[base + s_from[p]];
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < ITEMS; i++) {
            const uint32_t p = (uint32_t)i * BLOCK + threadIdx.x;
            if (p < cnt) out_v[base + p] = v[i];
        }
    }
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
        const uint32_t p = (uint32_t)i * BLOCK + threadIdx.x;
        if (p < cnt) out_k[base + p] = (OK)s_k[merge_slot<PAD>(p)];
    }
}

// One warp: how many of the first d outputs of merging the runs a[0, na) and b[0, nb) come from
// a (32 probes per round).
template <class K, class Comp>
TRTC_FORCEINLINE size_t merge_path_warp(const K* a, size_t na, const K* b, size_t nb, size_t d, Comp& comp) {
    size_t lo = d > nb ? d - nb : 0, hi = d < na ? d : na;
    while (lo < hi) {
        const size_t span = hi - lo;
        // probe offset of lane l: l for short spans, span * (l + 1) / 32 or so else (ascending,
        // the last one below span)
        const size_t step = span / 33 + 1;
        const size_t m = lo + (span <= 32 ? (size_t)lane_id() : step * lane_id() + step - 1);
        // is a[m] among the first d outputs?  (true for a prefix of the probes)
        bool left = false;
        if (m < hi) left = !(bool)comp(b[d - 1 - m], a[m]);
        const uint32_t c = (uint32_t)__popc(__ballot_sync(0xffffffffu, left));
        if (span <= 32) { lo += (size_t)c; break; }
        const size_t nhi = lo + step * c + step - 1;  // probe c, not left (or past hi)
        lo += step * c;                               // behind probe c - 1, left
        hi = nhi < hi ? nhi : hi;
        if (lo > hi) lo = hi;
    }
    return lo;
}

// Merges the sorted runs of `width` (a multiple of BLOCK * ITEMS) elements of in_k / in_v
// pairwise.
template <class K, class V, class OKV, class OVV, class Comp, bool HAS_VALS, int BLOCK, int ITEMS>
__global__ void __launch_bounds__(BLOCK) merge_level_kernel(const K* __restrict__ in_k, const V* __restrict__ in_v,
                                                            OKV out_k, OVV out_v, size_t n, size_t width, Comp comp) {
    constexpr uint32_t T = BLOCK * ITEMS;
    static_assert(BLOCK >= 64, "two searching warps");
    // 4-byte values beside 4-byte keys are staged with them; wider ones are gathered from the
    // runs at the end (two sequential streams)
    constexpr bool SV = HAS_VALS && sizeof(K) <= 4 && sizeof(V) <= 4;
    __shared__ __align__(16) K s_k[T + 1];
    // (bytes: aligned for 4-byte asynchronous copies whatever V's own alignment is, and without V's
    // constructor, which a shared variable may not have)
    __shared__ __align__(16) unsigned char s_vbytes[SV ? T * sizeof(V) : 16];
    V* const s_v = reinterpret_cast<V*>(s_vbytes);
    __shared__ __align__(16) unsigned short s_from[T];
    __shared__ size_t s_path[2];
    typedef typename remove_cvref<typename OKV::value_t>::type OK;
    const size_t out0 = (size_t)blockIdx.x * T;  // first output of the tile
    const size_t a0 = out0 & ~(2 * width - 1);   // width is a power of two
    const size_t mid = a0 + width < n ? a0 + width : n, end = a0 + 2 * width < n ? a0 + 2 * width : n;
    const size_t na = mid - a0, nb = end - mid, d0 = out0 - a0;
    const uint32_t cnt = (uint32_t)((end - out0) < (size_t)T ? (end - out0) : (size_t)T);
    const uint32_t warp = threadIdx.x >> 5;
    if (warp < 2) {
        const size_t r = merge_path_warp<K, Comp>(in_k + a0, na, in_k + mid, nb, d0 + (warp ? (size_t)cnt : 0), comp);
        if (lane_id() == 0) s_path[warp] = r;
    }
    __syncthreads();
    const size_t pa = s_path[0];
    size_t pe = s_path[1];
    {
        // 0 <= left part <= cnt, both parts inside their runs, whatever the comparator says
        const size_t dn = d0 + (size_t)cnt;
        const size_t low = dn > nb ? dn - nb : 0;
        const size_t lo = pa > low ? pa : low;
        const size_t hi = na < pa + (size_t)cnt ? na : pa + (size_t)cnt;
        pe = pe < lo ? lo : (pe > hi ? hi : pe);
    }
    const uint32_t ca = (uint32_t)(pe - pa);  // the tile: ca elements of the left run, then cnt - ca of the right
    // tile element p is in_k[ga + p] for p < ca, else in_k[gb + p]
    const size_t ga = a0 + pa, gb = mid + (d0 - pa) - (size_t)ca;
    auto body = [&](auto full_c) {
        constexpr bool FULL = decltype(full_c)::value;
        // all of the thread's keys and values in flight together, without registers
        const K* ka = in_k + ga + threadIdx.x;
        const K* kb = in_k + gb + threadIdx.x;
        const V* va = in_v + ga + threadIdx.x;
        const V* vb = in_v + gb + threadIdx.x;
#pragma unroll
        for (int i = 0; i < ITEMS; i++) {
            const uint32_t p = (uint32_t)i * BLOCK + threadIdx.x;
            if (FULL || p < cnt) {
                merge_copy_async(s_k + p, (p < ca ? ka : kb) + i * BLOCK);
                if constexpr (SV) merge_copy_async(s_v + p, (p < ca ? va : vb) + i * BLOCK);
            }
        }
        merge_copy_wait();
        __syncthreads();
        const uint32_t d = threadIdx.x * ITEMS;
        if (FULL || d < cnt) {
            unsigned short src[ITEMS];
            const uint32_t ta = merge_path_tile<K, Comp, false>(s_k, 0u, ca, ca, cnt - ca, d, comp);
            merge_serial<K, Comp, ITEMS, false, FULL>(s_k, ta, ca, ca + d - ta, cnt, comp, src);
            merge_store_from<ITEMS>(s_from + d, src);
        }
        __syncthreads();
        const size_t o = out0 + threadIdx.x;
#pragma unroll
        for (int i = 0; i < ITEMS; i++) {
            const uint32_t p = (uint32_t)i * BLOCK + threadIdx.x;
            if (FULL || p < cnt) {
                const uint32_t f = s_from[p];
                out_k[o + i * BLOCK] = (OK)s_k[f];
                if constexpr (SV) {
                    typedef typename remove_cvref<typename OVV::value_t>::type OV;
                    out_v[o + i * BLOCK] = (OV)s_v[f];
                }
            }
        }
        if constexpr (HAS_VALS && !SV) {
            typedef typename remove_cvref<typename OVV::value_t>::type OV;
            OV v[ITEMS];
#pragma unroll
            for (int i = 0; i < ITEMS; i++) {
                const uint32_t p = (uint32_t)i * BLOCK + threadIdx.x;
                if (FULL || p < cnt) {
                    const uint32_t f = s_from[p];
                    v[i] = (OV)in_v[(f < ca ? ga : gb) + (size_t)f];
                }
            }
#pragma unroll
            for (int i = 0; i < ITEMS; i++) {
                const uint32_t p = (uint32_t)i * BLOCK + threadIdx.x;
                if (FULL || p < cnt) out_v[o + i * BLOCK] = v[i];
            }
        }
    };
    if (cnt == T) body(MergeBool<true>()); else body(MergeBool<false>());
}

// out[out_off + i] = (out element type) in[in_off + i] for i < count, where count is n, or
// n - *tail_base when tail_base is given (partition tails whose length is known on device).
template <class InV, class OutV>
__global__ void copy_view_kernel(InV in, OutV out, size_t n, size_t in_off, size_t out_off,
                                 const unsigned long long* tail_base) {
    typedef typename remove_cvref<typename OutV::value_t>::type O;
    size_t count = n;
    size_t ooff = out_off;
    if (tail_base) {
        count = n - (size_t)*tail_base;
        ooff += (size_t)*tail_base;
    }
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (size_t)gridDim.x * blockDim.x)
        out[ooff + i] = (O)in[in_off + i];
}

}  // namespace trtc
