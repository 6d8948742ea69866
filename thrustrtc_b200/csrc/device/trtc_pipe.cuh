// trtc_pipe.cuh -- persistent tile pipeline: reduce_by_key and compaction in one pass.
//
// The reference reduces by key with a segmented scan of every element, a scan of the tail
// flags and a scatter (reduce.cpp:36-62), and compacts with a flag scan and a scatter
// (internal/general_copy_if.cpp:26-64).  Here a tile is read once, its segments are folded or its
// elements selected on chip, and only the results leave it.
//
// A CTA runs five roles, handed from one to the next through mbarriers, so that none waits for
// another's latency:
//   producer          takes tile tickets in order and brings each tile into one of S input
//                     stages by TMA bulk copies;
//   compute groups    (of 8 warps; tile k of the CTA is group k % G's) fold the tile, publish its
//                     aggregates, give the input stage back and stage the results in a ring;
//   await warps       wait for what the tile needs from earlier tiles: the number of results
//                     before it (and the running value of the segment that enters it);
//   store warps       write the staged results at their final place (a tile each).
// One CTA of the grid, the prefix CTA, scans what the tiles publish (half of its warps the counts,
// half the running values where there are any) and answers every tile with what precedes it.  Tickets are drawn in
// order by running CTAs, so a tile only ever waits for tiles that are under way.  A worker that runs
// draws until the end.  When none does (a long kernel of another stream leaves room for the prefix CTA
// only), calls that read a result back give up before the first tile and the host takes the general form;
// the scan, whose call has returned by then, does tiles in the prefix CTA.
//
// Every wait is bounded: a role whose wait expires records the error and leaves, the others
// follow (their waits see the error word), and the producer draws its remaining tickets so
// that the ticket counter is back at zero for the next call.
#pragma once
#include "trtc_compact.cuh"

namespace trtc {

enum : int {
    PIPE_COMPUTE = 8,   // warps of a compute group
    PIPE_STORE = 4,     // store warps
    PIPE_META = 16,     // tiles of a CTA between folding and stored, at most
    PIPE_ALONE = 1024   // polls (about 1 ms; workers draw within microseconds of their start) before the
                        // prefix CTA takes itself to be alone
};
template <int G> struct PipeShape {
    enum : int { WARPS = PIPE_COMPUTE * G + PIPE_STORE + 3, THREADS = WARPS * 32 };
};
enum : uint32_t { PIPE_END = 0xFFFFFFFFu };

// barrier `id` among `threads` threads; with a vote: true when any of them passes true
TRTC_FORCEINLINE void pipe_sync(uint32_t id, uint32_t threads) {
    asm volatile("barrier.cta.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
TRTC_FORCEINLINE bool pipe_any(uint32_t id, uint32_t threads, bool v) {
    uint32_t r;
    asm volatile("{\n .reg .pred p, q;\n setp.ne.u32 p, %3, 0;\n barrier.cta.red.or.pred q, %1, %2, p;\n selp.u32 %0, 1, 0, q;\n}\n"
                 : "=r"(r) : "r"(id), "r"(threads), "r"((uint32_t)v) : "memory");
    return r != 0;
}

// What a tile publishes (state 1, + 4 when it holds a segment head) and what the prefix CTA
// answers (state 2, + 4 when there is a value before the tile): one 64-bit word per tile for
// values of up to 4 bytes, else a value array per direction and a flag word.
template <class T>
TRTC_FORCEINLINE void pipe_put(const LookbackState& st, uint32_t tile, const T& v, uint32_t state) {
    const uint32_t fw = st.epoch8 + state;
    if constexpr (LbPack<T>::value) {
        st_relaxed(&st.packed[tile], ((unsigned long long)fw << 32) | (unsigned long long)lb_bits<T>(v));
    } else {
        reinterpret_cast<T*>((state & 2u) ? st.incl : st.agg)[tile] = v;
        st_release(&st.flags[tile], fw);
    }
}
// the state of a tile's word (0: not of this launch); v: its value where it travels in the word
template <class T>
TRTC_FORCEINLINE uint32_t pipe_peek(const LookbackState& st, uint32_t tile, T& v) {
    if constexpr (LbPack<T>::value) {
        const unsigned long long w = ld_relaxed(&st.packed[tile]);
        v = lb_value<T>((uint32_t)w);
        return lb_state((uint32_t)(w >> 32), st.epoch8);
    } else {
        return lb_state(ld_relaxed(&st.flags[tile]), st.epoch8);
    }
}
// the prefix CTA's answer for `tile` (0: not there yet)
template <class T>
TRTC_FORCEINLINE uint32_t pipe_answer(const LookbackState& st, uint32_t tile, T& v) {
    const uint32_t f = pipe_peek<T>(st, tile, v);
    if (!(f & 2u)) return 0u;
    if constexpr (!LbPack<T>::value) {
        fence_acq_rel();
        v = reinterpret_cast<const T*>(st.incl)[tile];
    }
    return f;
}
// One warp, lane m on bookkeeping slot m: passes every tile of the CTA on from agg to pref once
// take(m, tile) has found its answer; returns when all tiles before the end mark are passed on.
template <class Take>
TRTC_FORCEINLINE void pipe_await_slots(unsigned long long* agg, unsigned long long* pref, const uint32_t* m_tile,
                                       uint32_t* err, Take take) {
    const uint32_t m = lane_id();
    uint32_t k = m, tile = 0, passed = 0, spins = 0;
    bool have = false;
    while (true) {
        bool moved = false;
        if (m < (uint32_t)PIPE_META) {
            if (!have && mbar_test(&agg[m], (k / PIPE_META) & 1u)) {
                have = true;
                tile = *(volatile const uint32_t*)&m_tile[m];
            }
            if (have && tile != PIPE_END && take(m, tile)) {
                mbar_arrive(&pref[m]);
                have = false;
                k += PIPE_META;
                moved = true;
            }
        }
        const uint32_t now = (uint32_t)__popc(__ballot_sync(0xffffffffu, moved));
        passed += now;
        const uint32_t end = __reduce_min_sync(0xffffffffu, have && tile == PIPE_END ? k : 0xffffffffu);
        if (passed == end) return;
        if (now) spins = 0;
        else if (__any_sync(0xffffffffu, !spin_continue(spins, err))) {
            if (m == 0) report_error(err, TRTC_ERR_LOOKBACK_TIMEOUT);
            return;
        }
    }
}

// Alone before the first tile: takes all tickets, so that workers that come later leave at once, and
// reports ~0 as the call's result.  `gone` (shared memory, zero) tells the other half of the CTA, whose
// own PipeCancel has no result.
struct PipeCancel {
    unsigned long long* ctr;
    uint32_t tiles;
    volatile uint32_t* gone;
    unsigned long long* result;
    TRTC_FORCEINLINE bool now(uint32_t first, uint32_t spins) {
        if (!result) return *gone != 0u;
        const unsigned long long end = (unsigned long long)tiles + 1u;
        if (first > 0u || spins < (uint32_t)PIPE_ALONE || atomicCAS(ctr, 1ull, end) != 1ull) return false;
        if (gridDim.x == 1) atomicExch(ctr, 0ull);  // (no worker to draw the last ticket)
        *result = ~0ull;
        *gone = 1u;
        return true;
    }
    template <class T> TRTC_FORCEINLINE bool act(uint32_t, const T&, bool) { return false; }
};

// Alone at any tile: draws it (draw(tile): false when somebody else has) and does it (tile_alone).
template <class Draw, class Tile> struct PipeSolo {
    Draw draw;
    Tile tile_alone;
    uint32_t patience = PIPE_ALONE;
    TRTC_FORCEINLINE bool now(uint32_t first, uint32_t spins) {
        if (spins < patience) return false;
        const bool mine = draw(first);
        patience = mine ? 8u : (uint32_t)PIPE_ALONE;
        return mine;
    }
    template <class T> TRTC_FORCEINLINE bool act(uint32_t first, const T& run, bool run_h) {
        tile_alone(first, run, run_h);
        return true;
    }
};

// What the prefix CTA needs to do a tile itself, one element per thread of WARPS warps at a time (no
// stages: the prefix is known).  The elements of a chunk are those of its first threads.
// PipeRun: what a tile has come to before a chunk: its running value (when there is one), and whether no head
// stood in it so far.
template <class T> struct PipeRun {
    T v = T();
    bool has = false, open = true;
};
template <class T, int WARPS> struct PipeChunk {
    T v[WARPS];
    uint32_t has[WARPS], head[WARPS];
};
// inclusive segmented scan behind `run`, which moves on past the chunk; open: no head in the tile up to
// this thread's element
template <int WARPS, class T, class Op>
TRTC_FORCEINLINE T pipe_chunk_scan(T v, bool head, bool valid, Op& op, uint32_t warp, uint32_t bar,
                                   PipeChunk<T, WARPS>* s, PipeRun<T>& run, bool& open) {
    const uint32_t lane = lane_id(), le = lane == 31u ? 0xffffffffu : ((2u << lane) - 1u);
    const uint32_t vm = __ballot_sync(0xffffffffu, valid), hm = __ballot_sync(0xffffffffu, valid && head);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const T y = shfl_up_any(v, d);
        if (valid && lane >= (uint32_t)d) {
            const uint32_t win = le & ~((1u << (lane - (uint32_t)d + 1u)) - 1u);
            if ((hm & win) == 0u) v = (T)op(y, v);
        }
    }
    if (vm && lane == 31u - (uint32_t)__clz(vm)) s->v[warp] = v;
    if (lane == 0) {
        s->has[warp] = vm != 0u;
        s->head[warp] = hm != 0u;
    }
    pipe_sync(bar, WARPS * 32);
    open = false;
#pragma unroll 1
    for (uint32_t w = 0; w < (uint32_t)WARPS; w++) {
        if (w == warp) {
            if (valid && (hm & le) == 0u && run.has) v = (T)op(run.v, v);
            open = run.open && (hm & le) == 0u;
        }
        if (!s->has[w]) continue;
        run.v = (s->head[w] || !run.has) ? s->v[w] : (T)op(run.v, s->v[w]);
        run.has = true;
        run.open = run.open && !s->head[w];
    }
    pipe_sync(bar, WARPS * 32);  // s is free
    return v;
}

// Half of the prefix CTA: polls one tile per thread from the first unanswered one on, takes in the published
// ones that follow without a gap, scans them across the CTA and answers each with what precedes
// it (SEG: a segmented scan, a head discards what is before it).  Tiles then poll a single word
// of their own.  With a decoupled look-back by every tile instead (300 to 1200 warps polling up
// to 128 words a round, the frontier moving one window per round trip) the tiles of 50 M elements
// took 150 to 210 us where they take 88 us without any wait for prefixes.
// WARPS warps from warp0 on run one stream of values, published in st, answered in `answers` (the same
// words, or others); bar: a barrier of their own.
// alone: what to do while no other CTA runs (PipeCancel, or a kernel's own).  alone.now(first, spins), by one
// thread after a poll without progress: is it time?  Then alone.act(first, run, run_h), by all: false to leave.
template <class T, class Op, bool SEG, int WARPS, class Alone>
__device__ void pipe_prefix_scan(const LookbackState& st, const LookbackState& answers, uint32_t tiles, Op& op,
                                 unsigned long long* result, uint32_t warp0, uint32_t bar, Alone alone) {
    static_assert(WARPS <= 16, "one scan of 16 warps");
    __shared__ uint32_t s_lead[32], s_hd[32], s_has[32], s_taken;
    __shared__ T s_v[32], s_total;
    const uint32_t warp = (threadIdx.x >> 5) - warp0, lane = lane_id(), thread = warp * 32 + lane;
    uint32_t first = 0, spins = 0;  // first unanswered tile
    T run = T();                    // what precedes it
    bool run_h = false;
    if (thread < 32) s_lead[thread] = 0;
    const uint32_t le = lane == 31u ? 0xffffffffu : ((2u << lane) - 1u);  // lanes <= l
    while (first < tiles) {
        const uint32_t j = first + thread;
        uint32_t f = 0;
        T v = T();
        if (j < tiles) f = pipe_peek<T>(st, j, v);
        const uint32_t m = __ballot_sync(0xffffffffu, f != 0u);
        const uint32_t lead = m == 0xffffffffu ? 32u : (uint32_t)__ffs(~m) - 1u;  // ready without a gap
        if constexpr (!LbPack<T>::value) {
            fence_acq_rel();
            if (f) v = reinterpret_cast<const T*>(st.agg)[j];
        }
        // inclusive scan over the lanes before the gap (op only ever sees what was published: behind
        // the gap v is T(), or what an earlier call left in the word)
        const uint32_t hm = SEG ? __ballot_sync(0xffffffffu, (f & 4u) != 0u) : 0u;
        T vi = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const T vy = shfl_up_any(vi, d);
            if (lane >= (uint32_t)d && lane < lead) {
                const uint32_t win = le & ~((1u << (lane - (uint32_t)d + 1u)) - 1u);
                if ((hm & win) == 0u) vi = (T)op(vy, vi);
            }
        }
        const T ve = shfl_up_any(vi, 1);
        if (lane == (lead ? lead - 1u : 0u)) {
            s_lead[warp] = lead;
            s_v[warp] = vi;
            s_hd[warp] = lead && (hm & le) != 0u;
        }
        pipe_sync(bar, WARPS * 32);
        if (warp == 0) {
            // the same over the warps that are taken in: all before the first gap, and that one
            const uint32_t l = lane < (uint32_t)WARPS ? s_lead[lane] : 0u;
            const uint32_t fullm = __ballot_sync(0xffffffffu, l == 32u);
            const uint32_t nfull = (uint32_t)__ffs(~fullm) - 1u;  // warps without a gap, from warp 0 on
            const bool in = lane < nfull || (lane == nfull && l > 0u);
            const uint32_t inm = __ballot_sync(0xffffffffu, in);
            T w = in ? s_v[lane] : T();
            const uint32_t wh = __ballot_sync(0xffffffffu, in && s_hd[lane] != 0u);
#pragma unroll
            for (int d = 1; d < 16; d <<= 1) {
                const T y = shfl_up_any(w, d);
                if (lane >= (uint32_t)d && in) {
                    const uint32_t win = le & ~((1u << (lane - (uint32_t)d + 1u)) - 1u);
                    if ((wh & win) == 0u) w = (T)op(y, w);
                }
            }
            // what precedes the warp's first tile
            const T y = shfl_up_any(w, 1);
            const bool yhd = (wh & (le >> 1)) != 0u;
            const uint32_t nin = (uint32_t)__popc(inm);  // (lanes 0 to nin - 1)
            T pre = run;
            if (lane > 0 && in) pre = (yhd || !run_h) ? y : (T)op(run, y);
            s_v[lane] = pre;
            s_has[lane] = run_h || lane > 0 ? 1u : 0u;
            if (nin && lane == nin - 1u) s_total = ((wh & le) != 0u || !run_h) ? w : (T)op(run, w);
            const uint32_t t = __reduce_add_sync(0xffffffffu, in ? l : 0u);
            s_lead[lane] = in ? l : 0u;
            if (lane == 0) s_taken = t;
        }
        pipe_sync(bar, WARPS * 32);
        const uint32_t taken = s_taken;
        if (lane < s_lead[warp]) {
            T p = s_v[warp];
            bool ph = s_has[warp] != 0u;
            if (lane > 0) {
                p = ((hm & (le >> 1)) != 0u || !ph) ? ve : (T)op(p, ve);
                ph = true;
            }
            pipe_put<T>(answers, j, p, ph ? 6u : 2u);
        }
        if (taken) {
            run = s_total;
            run_h = true;
            spins = 0;
        }
        bool give_up = false, act = false;
        if (!taken) {
            give_up = !spin_continue(spins, st.err);
            act = thread == 0 && alone.now(first, spins);
        }
        if (pipe_any(bar, WARPS * 32, give_up || act)) {
            const bool fail = pipe_any(bar, WARPS * 32, give_up);
            if (fail) report_error(st.err, TRTC_ERR_LOOKBACK_TIMEOUT);
            if (fail || !alone.act(first, run, run_h)) return;
        }
        first += taken;
    }
    if constexpr (!SEG)
        if (result && thread == 0) *result = (unsigned long long)run;
}

// inclusive sums over the lanes, up to distance `lanes` / 2: the shuffle's own in-range predicate
// gates the addition
template <int LANES>
TRTC_FORCEINLINE uint32_t pipe_lane_sums(uint32_t v) {
#pragma unroll
    for (int d = 1; d < LANES; d <<= 1)
        asm volatile("{\n .reg .pred p;\n .reg .u32 t;\n shfl.sync.up.b32 t|p, %0, %1, 0, 0xffffffff;\n @p add.u32 %0, %0, t;\n}\n"
                     : "+r"(v) : "r"(d));
    return v;
}

// A parity wait tells a phase from its neighbours only, so a waiter has to be at most one phase behind
// or ahead.  Stage k % S is loaded for other groups in between where S is not a multiple of G, and
// loads complete in any order: "loaded" has a barrier per k % L, L a multiple of both, each always the
// same group's, which waits for every phase of it.
template <int S, int L> struct PipeBars {
    unsigned long long full[L];            // tile loaded (producer, and its bulk copies)
    unsigned long long empty[S];           // input stage read (compute warps)
    unsigned long long agg[PIPE_META];     // aggregates published (compute)
    unsigned long long comp[PIPE_META];    // results staged (compute warps)
    unsigned long long pref[PIPE_META];    // prefixes known (await warps)
    unsigned long long done[PIPE_META];    // results written (store warp)
    TRTC_FORCEINLINE void init(uint32_t await_warps) {
        for (int s = 0; s < L; s++) mbar_init(&full[s], 1u);
        for (int s = 0; s < S; s++) mbar_init(&empty[s], (uint32_t)PIPE_COMPUTE);
        for (int m = 0; m < PIPE_META; m++) {
            mbar_init(&agg[m], 1u);
            mbar_init(&comp[m], (uint32_t)PIPE_COMPUTE);
            mbar_init(&pref[m], await_warps);
            mbar_init(&done[m], 1u);
        }
        mbar_init_fence();
    }
};

// ITEMS consecutive elements of shared memory into registers, in 16-byte loads where they fill
// whole ones (an odd number of them per thread: no bank conflicts)
template <class T, int ITEMS>
TRTC_FORCEINLINE void pipe_load_run(const T* s, T (&v)[ITEMS]) {
    if constexpr ((sizeof(T) == 4 || sizeof(T) == 8) && sizeof(T) * ITEMS % 16 == 0) {
        union U { uint4 q[sizeof(T) * ITEMS / 16]; T t[ITEMS]; TRTC_FORCEINLINE U() {} } u;
#pragma unroll
        for (int i = 0; i < (int)(sizeof(T) * ITEMS / 16); i++) u.q[i] = reinterpret_cast<const uint4*>(s)[i];
#pragma unroll
        for (int i = 0; i < ITEMS; i++) v[i] = u.t[i];
    } else {
#pragma unroll
        for (int i = 0; i < ITEMS; i++) v[i] = s[i];
    }
}

// The producer: draws tickets (the first, `t`, is already drawn; ticket t > 0 is tile t - 1) and has
// issue(stage, tile, barrier) start the tile's bulk copies, or not (false: the compute group loads
// the tile itself); after the last tile one stage per group carries the end mark.  A draw's round
// trip (0.4 us) and the issue (0.3 us) bound a CTA's tile rate where a tile costs less than that.
template <int G, int S, int L, class Issue>
TRTC_FORCEINLINE void pipe_produce(PipeBars<S, L>& bars, const LookbackState& st, uint32_t tiles, unsigned long long t,
                                   uint32_t* s_tile, uint32_t* s_bulk, Issue issue) {
    static_assert(S >= G, "the end reaches every group");
    const unsigned long long last = (unsigned long long)tiles + gridDim.x - 1;
    uint32_t ends = 0;
    for (uint32_t k = 0;; k++) {
        const uint32_t s = k % S;
        if (k > 0 && ends == 0) t = atomicAdd(st.tile_ctr, 1ull);
        if (ends == 0 && t == last) atomicExch(st.tile_ctr, 0ull);  // every ticket is taken
        const bool ok = k < S || mbar_wait_bounded(&bars.empty[s], (k / S + 1u) & 1u, st.err);
        if (!ok) {
            report_error(st.err, TRTC_ERR_LOOKBACK_TIMEOUT);
            while (t <= (unsigned long long)tiles)
                if ((t = atomicAdd(st.tile_ctr, 1ull)) == last) atomicExch(st.tile_ctr, 0ull);
            // copies still under way write this CTA's shared memory
            for (uint32_t q = k - S; q < k; q++) mbar_wait_bounded(&bars.full[q % L], (q / L) & 1u, nullptr);
            return;
        }
        if (t > (unsigned long long)tiles) {
            s_tile[s] = PIPE_END;
            mbar_arrive(&bars.full[k % L]);
            if (++ends == (uint32_t)G) return;
            continue;
        }
        const uint32_t tile = (uint32_t)t - 1u;
        s_tile[s] = tile;
        s_bulk[s] = 0u;
        if (!issue(s, tile, &bars.full[k % L])) mbar_arrive(&bars.full[k % L]);
    }
}
// The store warps' wait for tile k of the CTA: 0 when it may be written, 1 at the end (m_last, the
// CTA's number of tiles once known, is not above k), 2 when the wait ran out.
template <int S, int L>
TRTC_FORCEINLINE int pipe_store_wait(PipeBars<S, L>& bars, uint32_t k, const uint32_t* m_last, uint32_t* err) {
    const uint32_t m = k % PIPE_META, ph = (k / PIPE_META) & 1u;
    uint32_t spins = 0;
    int r = 0;
    while (!mbar_try_wait(&bars.pref[m], ph)) {
        if (*(volatile const uint32_t*)m_last <= k) { r = 1; break; }
        if (!spin_continue(spins, err)) { r = 2; break; }
    }
    if (r == 0 && !mbar_wait_bounded(&bars.comp[m], ph, err)) r = 2;
    if (__any_sync(0xffffffffu, r == 2)) {
        if (lane_id() == 0) report_error(err, TRTC_ERR_LOOKBACK_TIMEOUT);
        return 2;
    }
    return __any_sync(0xffffffffu, r == 1) ? 1 : 0;
}

// element sizes whose tiles are brought in by bulk copies (when contiguous and aligned)
template <class T> struct PipeBulk {
    static constexpr bool value = sizeof(T) == 1 || sizeof(T) == 2 || sizeof(T) == 4 || sizeof(T) == 8;
};

// a staged result (one shared-memory access where the sizes allow)
template <class K, class T> struct RbkAlign {
    static constexpr int value = sizeof(K) == 4 && sizeof(T) == 4 ? 8
                                 : (sizeof(K) == 8 || sizeof(T) == 8) && sizeof(K) + sizeof(T) > 8 && sizeof(K) + sizeof(T) <= 16
                                     ? 16 : (alignof(K) > alignof(T) ? (int)alignof(K) : (int)alignof(T));
};
template <class K, class T> struct alignas(RbkAlign<K, T>::value) RbkResult {
    K k;
    T v;
};

// Shared memory of the reduce_by_key pipeline: S input stages (keys with one 16-byte halo on both
// sides, or one element where 16 bytes are not whole elements; then the values) and the ring of
// staged results: C results, and room for a tile's behind it, so that the results of a tile that
// starts before the ring's end need not wrap.
template <class K, class E, class T, int ITEMS, int S, int C> struct RbkSmem {
    static constexpr int TILE = PIPE_COMPUTE * 32 * ITEMS;
    static_assert(C >= TILE, "a tile's results fit the ring");
    static constexpr int HALO = PipeBulk<K>::value ? 16 / (int)sizeof(K) : 1;
    static constexpr size_t KEY_BYTES = ((size_t)(TILE + 2 * HALO) * sizeof(K) + 15) / 16 * 16;
    static constexpr size_t STAGE = KEY_BYTES + ((size_t)TILE * sizeof(E) + 15) / 16 * 16;
    static constexpr size_t RING = S * STAGE;
    static constexpr size_t BYTES = RING + (size_t)(C + TILE) * sizeof(RbkResult<K, T>);
    static_assert(BYTES <= PIPE_SMEM, "the launch's shared memory");
};

// B200, 50,000,011 int32 keys in runs of mean 32 with float sums: 85-90 us per launch (4.4 TB/s,
// 0.70 of the measured copy rate; segmented scan + tail compaction: 156 + 157 us); runs of 3:
// 142 us, one run: 81 us.  DRAM at 4.6 TB/s, issue 55 % busy, the ALU pipe 49 % (ncu): the fold of a tile
// costs about 40 instructions per element.  Runs of one, 50 M: 467 us per call, bound by the ring, which
// holds 1.5 tiles of results (two stages instead of three 275 us there, runs of 32 10 % slower).  Tiles of 20 elements per thread in 2 groups and 3 stages:
// 87 us; 12 elements, 3 groups, 6 stages: 95 us; 12, 2, 6: 106 us (the per-tile part of the fold
// spreads over fewer elements).  Two CTAs per SM of one group each, 12 elements: 128 us.
//
// Segments continue from i - 1 to i while pred(key[i-1], key[i]); the key of a segment's last
// element goes to out_k, op over its values (converted to T) to out_v, both in order; the
// number of segments to *st.result.  st: words of the counts, st2: of the running values.  The
// outputs do not overlap the inputs.
template <class KV, class VV, class OKV, class OVV, class T, class Pred, class Op, int G, int ITEMS, int S, int C>
__global__ void __launch_bounds__(PipeShape<G>::THREADS, 1) rbk_pipe_kernel(KV keys, VV vals, OKV out_k, OVV out_v, size_t n,
                                                                   uint32_t tiles, Pred pred, Op op, LookbackState st,
                                                                   LookbackState st2) {
    typedef typename remove_cvref<typename KV::value_t>::type K;
    typedef typename remove_cvref<typename VV::value_t>::type E;
    typedef RbkSmem<K, E, T, ITEMS, S, C> SM;
    constexpr uint32_t TILE = SM::TILE;
    constexpr int HALO = SM::HALO;
    static_assert(ITEMS < 32, "head mask");
    constexpr uint32_t OWN = (1u << ITEMS) - 1u;
    constexpr bool KTMA = ViewTraits<KV>::contiguous && PipeBulk<K>::value;
    constexpr bool VTMA = ViewTraits<VV>::contiguous && PipeBulk<E>::value;
    extern __shared__ __align__(16) unsigned char pipe_smem[];
    constexpr int L = S % G == 0 ? S : S * G;
    __shared__ PipeBars<S, L> bars;
    __shared__ uint32_t s_tile[S], s_bulk[S];                     // per input stage
    __shared__ uint32_t m_tile[PIPE_META], m_cnt[PIPE_META];      // per tile under way: its results,
    __shared__ uint32_t m_start[PIPE_META], m_base[PIPE_META];    // their place in the ring and in the output,
    __shared__ uint32_t m_open[PIPE_META], m_carry_h[PIPE_META];  // whether a segment enters it, and its value
    __shared__ T m_carry[PIPE_META];
    // the ring position behind a tile's results; kept for 2 x PIPE_META tiles, so that a group
    // still reads it while another takes the tile's slot for a later tile
    __shared__ uint32_t m_end[2 * PIPE_META], m_stored[2 * PIPE_META];  // (m_stored: tile + 1 once stored)
    __shared__ T s_wtot[2 * G][PIPE_COMPUTE];
    __shared__ __align__(16) uint32_t s_wcnt[2 * G][PIPE_COMPUTE];  // results of the warp's elements, bit 31: holds a head
    __shared__ uint32_t m_last;  // the CTA's number of tiles, once known
    __shared__ uint32_t s_gone;  // (prefix CTA)
    __shared__ unsigned long long s_first;

    const uint32_t warp = threadIdx.x >> 5, lane = lane_id();
    auto skey = [&](uint32_t s) -> K* { return reinterpret_cast<K*>(pipe_smem + s * SM::STAGE) + HALO; };
    auto sval = [&](uint32_t s) -> E* { return reinterpret_cast<E*>(pipe_smem + s * SM::STAGE + SM::KEY_BYTES); };
    RbkResult<K, T>* ring = reinterpret_cast<RbkResult<K, T>*>(pipe_smem + SM::RING);
    if (threadIdx.x == 0) bars.init(2u);
    if (threadIdx.x == 0) m_last = 0xFFFFFFFFu;
    if (threadIdx.x == 0) s_gone = 0u;
    if (threadIdx.x < 2 * PIPE_META) m_stored[threadIdx.x] = 0;
    // tickets: the first one makes its CTA the prefix CTA (running before any tile can wait for it),
    // ticket t > 0 is tile t - 1; every other CTA draws until it holds one past the last tile
    if (threadIdx.x == 0) s_first = atomicAdd(st.tile_ctr, 1ull);
    __syncthreads();
    if (s_first == 0) {
        constexpr int HALF = PipeShape<G>::WARPS / 2;
        Plus plus;
        unsigned long long* result = reinterpret_cast<unsigned long long*>(st.result);
        if (warp < HALF)
            pipe_prefix_scan<uint32_t, Plus, false, HALF>(st, st, tiles, plus, result, 0u, 1u,
                                                          PipeCancel{st.tile_ctr, tiles, &s_gone, result});
        else if (warp < 2 * HALF)
            pipe_prefix_scan<T, Op, true, HALF>(st2, st2, tiles, op, nullptr, HALF, 2u,
                                                PipeCancel{st.tile_ctr, tiles, &s_gone, nullptr});
        return;
    }
    constexpr uint32_t GT = PIPE_COMPUTE * 32;  // threads of a group

    if (warp < PIPE_COMPUTE * G) {
        // ------------------------------------------------------------ compute
        const uint32_t g = warp / PIPE_COMPUTE, gw = warp % PIPE_COMPUTE, gt = threadIdx.x % GT, bar = 1u + g;
        const uint32_t t0 = gt * ITEMS;
        uint32_t tail = 0, oldest = 0;  // ring position of the first tile not known to be stored
        for (uint32_t k = g;; k += G) {
            const uint32_t s = k % S, m = k % PIPE_META, b = (k / G % 2u) * G + g;
            bool fail = !mbar_wait_bounded(&bars.full[k % L], (k / L) & 1u, st.err);
            // the tile's bookkeeping slot is free again
            if (!fail && k >= (uint32_t)PIPE_META)
                fail = !mbar_wait_bounded(&bars.done[m], (k / PIPE_META + 1u) & 1u, st.err);
            if (fail) report_error(st.err, TRTC_ERR_LOOKBACK_TIMEOUT);
            if (pipe_any(bar, GT, fail)) return;
            const uint32_t tile = s_tile[s];
            if (gt == 0) m_tile[m] = tile;
            if (tile == PIPE_END) {
                if (gt == 0) {
                    atomicMin(&m_last, k);
                    mbar_arrive(&bars.agg[m]);
                }
                return;
            }
            const size_t base = (size_t)tile * TILE;
            const bool bulk = s_bulk[s] != 0;
            const uint32_t cnt = (n - base) < (size_t)TILE ? (uint32_t)(n - base) : TILE;
            K* kp = skey(s);
            E* vp = sval(s);
            if (!bulk) {
                for (uint32_t i = gt; i < cnt; i += GT) {
                    kp[i] = (K)keys[base + i];
                    vp[i] = (E)vals[base + i];
                }
                if (gt == 0 && base > 0) kp[-1] = (K)keys[base - 1];
                if (base + cnt < n) {
                    if (gt == 1) kp[cnt] = (K)keys[base + cnt];
                } else {
                    // no key behind the last: itself stands in (see tile 0)
                    const K last = (K)keys[n - 1];
                    for (uint32_t i = cnt + gt; i <= TILE; i += GT) kp[i] = last;
                }
            } else if (!VTMA) {
                for (uint32_t i = gt; i < TILE; i += GT) vp[i] = (E)vals[base + i];
            }
            // A user's predicate may index by the keys, so it only ever sees keys of the array: where a
            // neighbour is missing (its answer is not used) the key itself is put in the stage.  Tests
            // around the calls instead split the fold's straight line: 50 M elements 99.9 us per call, this way 95.8.
            if (tile == 0 && gt == 0) kp[-1] = (K)keys[0];
            if (!bulk || !VTMA || tile == 0) {
                // these writes come before a later bulk copy into the stage
                smem_proxy_fence();
                pipe_sync(bar, GT);
            }
            K kk[ITEMS];
            T x[ITEMS];
            pipe_load_run<K, ITEMS>(kp + t0, kk);
            {
                E e[ITEMS];
                pipe_load_run<E, ITEMS>(vp + t0, e);
#pragma unroll
                for (int j = 0; j < ITEMS; j++) x[j] = (T)e[j];
            }
            K prevk = shfl_up_any(kk[ITEMS - 1], 1), nextk = shfl_down_any(kk[0], 1);
            if (lane == 0) prevk = kp[(int)t0 - 1];
            if (lane == 31) nextk = kp[t0 + ITEMS];
            // the warp is done with the input stage
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars.empty[s]);
            // bit j: element j starts a segment (elements past the end count as heads)
            uint32_t hd = 0;
#pragma unroll
            for (int j = 0; j <= ITEMS; j++) {
                const K before = j == 0 ? prevk : kk[j > 0 ? j - 1 : 0];
                const K cur = j == ITEMS ? nextk : kk[j < ITEMS ? j : 0];
                if (!(bool)pred(before, cur)) hd |= 1u << j;
            }
            uint32_t left = ITEMS + 1u;  // this thread's elements (of the last tile)
            if (!bulk) {
                left = cnt > t0 ? cnt - t0 : 0u;
                if (base + cnt >= n && left <= (uint32_t)ITEMS) hd |= 0xffffffffu << left;
            }
            if (tile == 0 && gt == 0) hd |= 1u;
            // element j ends a segment when j + 1 starts one
            uint32_t tails = (hd >> 1) & OWN;
            if (left < (uint32_t)ITEMS) tails &= (1u << left) - 1u;
            // running values from the lane's first element or the last head on; the one after
            // its last head enters a segmented scan over the lanes.  Only the segment that enters
            // the lane (up to its first tail) lacks what precedes the lane.
#pragma unroll
            for (int j = 1; j < ITEMS; j++)
                if (!((hd >> j) & 1u)) x[j] = (T)op(x[j - 1], x[j]);
            const uint32_t hm = __ballot_sync(0xffffffffu, (hd & OWN) != 0u);
            const uint32_t le = lane == 31u ? 0xffffffffu : ((2u << lane) - 1u);  // lanes <= l
            const uint32_t mine = (uint32_t)__popc(tails);
            const uint32_t c = pipe_lane_sums<32>(mine);
            // a lane takes in the lanes down to the nearest one that holds a head
            const uint32_t dist = (hm & le) ? lane - (31u - (uint32_t)__clz(hm & le)) : lane;
            T inc = x[ITEMS - 1];
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const T y = shfl_up_any(inc, d);
                if ((uint32_t)d <= dist) inc = (T)op(y, inc);
            }
            const T ex = shfl_up_any(inc, 1);
            const bool exhd = (hm & (le >> 1)) != 0u;  // a head in lanes < l
            if (lane == 31) {
                s_wtot[b][gw] = inc;
                s_wcnt[b][gw] = c | (hm ? 0x80000000u : 0u);
            }
            pipe_sync(bar, GT);
            // the warps before this one: results, running value; the tile's results
            const uint32_t wc = lane < (uint32_t)PIPE_COMPUTE ? s_wcnt[b][lane] : 0u;
            const uint32_t whd = __ballot_sync(0xffffffffu, (wc >> 31) != 0u) & ((1u << gw) - 1u);  // holding heads
            const uint32_t wsum = pipe_lane_sums<PIPE_COMPUTE>(wc & 0x7fffffffu);
            const uint32_t total = __shfl_sync(0xffffffffu, wsum, PIPE_COMPUTE - 1);
            uint32_t pos = __shfl_sync(0xffffffffu, wsum - (wc & 0x7fffffffu), gw);
            T run = T();
            const bool run_hd = whd != 0u;
            bool run_h = gw > 0u;
            if (gw > 0u) {
                uint32_t w = run_hd ? 31u - (uint32_t)__clz(whd) : 0u;
                run = s_wtot[b][w];
#pragma unroll 1
                for (w++; w < gw; w++) run = (T)op(run, s_wtot[b][w]);
            }
            if (gw == PIPE_COMPUTE - 1 && lane == 31) {
                // the tile's aggregates
                const T agg = (!run_h || hm) ? inc : (T)op(run, inc);
                pipe_put<uint32_t>(st, tile, total, 1u);
                pipe_put<T>(st2, tile, agg, run_hd || hm != 0u ? 5u : 1u);
            }
            // the results' place in the ring: behind those of the CTA's tile before
            uint32_t head = 0;
            if (k > 0) {
                const uint32_t pm = (k - 1u) % PIPE_META;
                if (!mbar_wait_bounded(&bars.agg[pm], ((k - 1u) / PIPE_META) & 1u, st.err))
                    report_error(st.err, TRTC_ERR_LOOKBACK_TIMEOUT);
                head = m_end[(k - 1u) % (2 * PIPE_META)];
            }
            // every tile up to k - PIPE_META is stored: this one waited for the last of them, and the
            // tile before (whose aggregates it has seen) for the others
            if (k >= (uint32_t)PIPE_META && oldest <= k - PIPE_META) {
                oldest = k - PIPE_META + 1u;
                tail = m_end[(oldest - 1u) % (2 * PIPE_META)];
            }
            if (gw == PIPE_COMPUTE - 1 && lane == 31) {
                m_cnt[m] = total;
                m_start[m] = head % (uint32_t)C;
                m_end[k % (2 * PIPE_META)] = head + total;
                mbar_arrive(&bars.agg[m]);
            }
            if (gt == 0) m_open[m] = (hd & 1u) ? 0u : 1u;
            // room for the results in the ring
            for (uint32_t spins = 0; head + total - tail > (uint32_t)C;) {
                if (*(volatile uint32_t*)&m_stored[oldest % (2 * PIPE_META)] == oldest + 1u) {
                    tail = m_end[oldest % (2 * PIPE_META)];
                    oldest++;
                } else if (!spin_continue(spins, st.err)) {
                    report_error(st.err, TRTC_ERR_LOOKBACK_TIMEOUT);
                    break;
                }
            }
            {
                RbkResult<K, T>* r = ring + head % (uint32_t)C + pos + (c - mine);
                if (tails && !(hd & 1u)) {
                    // the segment that enters the lane: its first tail gets what precedes the lane
                    if (lane > 0) {
                        run = (exhd || !run_h) ? ex : (T)op(run, ex);
                        run_h = true;
                    }
                    const uint32_t first = tails & (0u - tails);
#pragma unroll
                    for (int j = 0; j < ITEMS; j++)
                        if (run_h && (first >> j) & 1u) x[j] = (T)op(run, x[j]);
                }
#pragma unroll
                for (int j = 0; j < ITEMS; j++) {
                    if ((tails >> j) & 1u) {
                        RbkResult<K, T> e;
                        e.k = kk[j];
                        e.v = x[j];
                        *r = e;
                        r++;
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars.comp[m]);
        }
    } else if (warp < PIPE_COMPUTE * G + PIPE_STORE) {
        // ------------------------------------------------------------ store
        const size_t ok_n = out_k.size(), ov_n = out_v.size();
        for (uint32_t k = warp - PIPE_COMPUTE * G;; k += PIPE_STORE) {
            const uint32_t m = k % PIPE_META;
            if (pipe_store_wait<S, L>(bars, k, &m_last, st.err)) return;
            const uint32_t cnt = m_cnt[m], start = m_start[m];
            const size_t base = m_base[m];
            const bool enters = m_open[m] && m_carry_h[m];  // the first result's segment began earlier
            const bool inside = base + cnt <= ok_n && base + cnt <= ov_n;
#pragma unroll 4
            for (uint32_t i = lane; i < cnt; i += 32) {
                const RbkResult<K, T> r = ring[start + i];
                const size_t o = base + i;
                if (inside || o < ok_n) out_k[o] = r.k;
                if (inside || o < ov_n) out_v[o] = (i == 0 && enters) ? (T)op(m_carry[m], r.v) : r.v;
            }
            __syncwarp();
            if (lane == 0) {
                __threadfence_block();
                *(volatile uint32_t*)&m_stored[k % (2 * PIPE_META)] = k + 1u;
                mbar_arrive(&bars.done[m]);
            }
        }
    } else if (warp < PIPE_COMPUTE * G + PIPE_STORE + 2) {
        // ------------------------------------------------------------ await (counts, running values)
        // lane m looks after bookkeeping slot m, so the answers of all tiles under way are polled
        // together (one after the other, a round trip each bounded the CTA's tile rate)
        const bool counts = warp == PIPE_COMPUTE * G + PIPE_STORE;
        pipe_await_slots(bars.agg, bars.pref, m_tile, st.err, [&](uint32_t m, uint32_t tile) -> bool {
            if (counts) {
                uint32_t pre = 0;
                if (!pipe_answer<uint32_t>(st, tile, pre)) return false;
                m_base[m] = pre;
            } else {
                T v = T();
                const uint32_t f = pipe_answer<T>(st2, tile, v);
                if (!f) return false;
                m_carry[m] = v;
                m_carry_h[m] = (f & 4u) ? 1u : 0u;
            }
            return true;
        });
    } else if (warp == PIPE_COMPUTE * G + PIPE_STORE + 2 && lane == 0) {
        // ------------------------------------------------------------ producer
        bool aligned = KTMA;
        if constexpr (KTMA) aligned = aligned && (reinterpret_cast<size_t>(keys._data) & 15u) == 0;
        if constexpr (VTMA) aligned = aligned && (reinterpret_cast<size_t>(vals._data) & 15u) == 0;
        pipe_produce<G, S, L>(bars, st, tiles, s_first, s_tile, s_bulk, [&](uint32_t s, uint32_t tile, unsigned long long* full) -> bool {
            const size_t base = (size_t)tile * TILE;
            if (!aligned || base + TILE + HALO > n) return false;
            if constexpr (KTMA) {
                const uint32_t lead = base > 0 ? (uint32_t)HALO : 0u;
                const uint32_t kb = (TILE + HALO + lead) * (uint32_t)sizeof(K);
                const uint32_t vb = VTMA ? TILE * (uint32_t)sizeof(E) : 0u;
                s_bulk[s] = 1u;
                mbar_arrive_expect(full, kb + vb);
                bulk_load_g2s_more(skey(s) - (int)lead, keys._data + base - lead, kb, full);
                if constexpr (VTMA) bulk_load_g2s_more(sval(s), vals._data + base, vb, full);
            }
            return true;
        });
    }
}

// ---------------------------------------------------------------- compaction
// Shared memory of the compaction pipeline: S input stages (the tile with a 16-byte lead, which
// holds the element before it) and the ring of selected (and rejected) elements, as above.
// Shapes: 3 groups, tiles of 20 KB (20 elements of 4 bytes, 10 of 8 per thread: 5 times 16 bytes, an odd
// number, so that the threads' 16-byte shared-memory loads do not share banks), 3 stages, the rest of
// 220 KB for the ring.  B200, 100 M int32, 50 / 90 / 100 % kept, us per launch: 3 groups, 20 elements, 3
// stages 124 / 173 / 183, 4 stages 121 / 187 / 198 (a smaller ring), 2 groups 3 stages 129 / 174 / 186,
// 2 groups 2 stages 136 / 167 / 175, 12 elements, 3 groups, 4 stages 154 / 169 / 175.  With few kept a
// CTA's rate of tickets and issues bounds it (0.73 us per tile), with half kept HBM (5.0 TB/s), with all
// kept the room for results that wait for their place (4 to 6 us from publication to answer).
template <class E> struct CpipeShape {
    static constexpr int G = 3, ITEMS = 80 / (int)sizeof(E), S = 3;
    static constexpr int TILE = PIPE_COMPUTE * 32 * ITEMS;
    static constexpr int RING = (((int)PIPE_SMEM - S * (TILE * (int)sizeof(E) + 16)) / (int)sizeof(E) - TILE) / 16 * 16;
    static constexpr size_t SMEM = S * ((size_t)TILE * sizeof(E) + 16) + (size_t)(RING + TILE) * sizeof(E);
};
template <class E, int ITEMS, int S> struct CpipeSmem {
    static constexpr int TILE = PIPE_COMPUTE * 32 * ITEMS;
    static constexpr int LEAD = 16 / (int)sizeof(E);
    static constexpr size_t STAGE = (size_t)(TILE + LEAD) * sizeof(E);
    static constexpr size_t RING = S * STAGE;
    static constexpr size_t bytes(size_t ring) { return RING + (ring + TILE) * sizeof(E); }
};

// Stable compaction of a contiguous array of 4- or 8-byte elements: elements selected by MODE
// (CM_PRED, CM_NOT_EQUAL, CM_NOT_PRED, CM_UNIQUE, CM_UNIQUE_PRED) go to out, the rejected ones of
// a partition to out_false, both in order; the number selected to *st.result.  The outputs do not
// overlap the input.  C: ring size in elements.
template <int MODE, bool PARTITION, class E, class Pred, class ValT, class OutV, class FalseV, int G, int ITEMS, int S, int C>
__global__ void __launch_bounds__(PipeShape<G>::THREADS, 1) compact_pipe_kernel(const E* in, Pred pred, ValT value, OutV out,
                                                                               FalseV out_false, size_t n, uint32_t tiles,
                                                                               LookbackState st) {
    typedef CpipeSmem<E, ITEMS, S> SM;
    constexpr uint32_t TILE = SM::TILE;
    constexpr bool NEIGH = MODE == CM_UNIQUE || MODE == CM_UNIQUE_PRED;
    static_assert(ITEMS < 32 && C >= (int)TILE, "selection mask; a tile's elements fit the ring");
    static_assert(SM::bytes(C) <= PIPE_SMEM, "the launch's shared memory");
    extern __shared__ __align__(16) unsigned char pipe_smem[];
    constexpr int L = S % G == 0 ? S : S * G;
    __shared__ PipeBars<S, L> bars;
    __shared__ uint32_t s_tile[S], s_bulk[S];
    __shared__ uint32_t m_tile[PIPE_META], m_cnt[PIPE_META], m_all[PIPE_META], m_start[PIPE_META], m_base[PIPE_META];
    __shared__ uint32_t m_end[2 * PIPE_META], m_stored[2 * PIPE_META];  // as in rbk_pipe_kernel
    __shared__ uint32_t s_wcnt[2 * G][PIPE_COMPUTE];
    __shared__ uint32_t m_last;
    __shared__ uint32_t s_gone;  // (prefix CTA)
    __shared__ unsigned long long s_first;

    const uint32_t warp = threadIdx.x >> 5, lane = lane_id();
    auto stage = [&](uint32_t s) -> E* { return reinterpret_cast<E*>(pipe_smem + s * SM::STAGE) + SM::LEAD; };
    E* ring = reinterpret_cast<E*>(pipe_smem + SM::RING);
    if (threadIdx.x == 0) {
        bars.init(1u);
        m_last = 0xFFFFFFFFu;
        s_gone = 0u;
        s_first = atomicAdd(st.tile_ctr, 1ull);
    }
    if (threadIdx.x < 2 * PIPE_META) m_stored[threadIdx.x] = 0;
    __syncthreads();
    if (s_first == 0) {
        constexpr int HALF = PipeShape<G>::WARPS / 2;
        Plus plus;
        unsigned long long* result = reinterpret_cast<unsigned long long*>(st.result);
        if (warp < HALF)
            pipe_prefix_scan<uint32_t, Plus, false, HALF>(st, st, tiles, plus, result, 0u, 1u,
                                                          PipeCancel{st.tile_ctr, tiles, &s_gone, result});
        return;
    }
    constexpr uint32_t GT = PIPE_COMPUTE * 32;  // threads of a group

    if (warp < PIPE_COMPUTE * G) {
        // ------------------------------------------------------------ compute
        const uint32_t g = warp / PIPE_COMPUTE, gw = warp % PIPE_COMPUTE, gt = threadIdx.x % GT, bar = 1u + g;
        const uint32_t t0 = gt * ITEMS;
        uint32_t tail = 0, oldest = 0;
        for (uint32_t k = g;; k += G) {
            const uint32_t s = k % S, m = k % PIPE_META, b = (k / G % 2u) * G + g;
            bool fail = !mbar_wait_bounded(&bars.full[k % L], (k / L) & 1u, st.err);
            if (!fail && k >= (uint32_t)PIPE_META)
                fail = !mbar_wait_bounded(&bars.done[m], (k / PIPE_META + 1u) & 1u, st.err);
            if (fail) report_error(st.err, TRTC_ERR_LOOKBACK_TIMEOUT);
            if (pipe_any(bar, GT, fail)) return;
            const uint32_t tile = s_tile[s];
            if (gt == 0) m_tile[m] = tile;
            if (tile == PIPE_END) {
                if (gt == 0) {
                    atomicMin(&m_last, k);
                    mbar_arrive(&bars.agg[m]);
                }
                return;
            }
            const size_t base = (size_t)tile * TILE;
            const uint32_t cnt = (n - base) < (size_t)TILE ? (uint32_t)(n - base) : TILE;
            E* p = stage(s);
            if (!s_bulk[s]) {
                for (uint32_t i = gt; i < cnt; i += GT) p[i] = in[base + i];
                if (NEIGH && gt == 0 && base > 0) p[-1] = in[base - 1];
                // these writes come before a later bulk copy into the stage
                smem_proxy_fence();
                pipe_sync(bar, GT);
            }
            E x[ITEMS];
            pipe_load_run<E, ITEMS>(p + t0, x);
            const uint32_t left = cnt > t0 ? cnt - t0 : 0u;  // this thread's elements
            auto test = [&](const E& v, const E& prev) -> bool {
                if constexpr (MODE == CM_PRED) return (bool)pred(v);
                else if constexpr (MODE == CM_NOT_EQUAL) return !(v == value);
                else if constexpr (MODE == CM_NOT_PRED) return !(bool)pred(v);
                else if constexpr (MODE == CM_UNIQUE) return v != prev;
                else return !(bool)pred(v, prev);
            };
            // A user's predicate is called on elements of the array only: it may index by its argument.
            // The last tile, and tile 0 where the neighbour is tested, take a loop over what there is; the
            // tiles between, all of whose elements (and neighbours) exist, an unrolled one without tests.
            const bool whole = cnt == TILE && !(NEIGH && tile == 0);
            uint32_t sel = 0;
            if (!whole) {
                const uint32_t end = left < (uint32_t)ITEMS ? left : (uint32_t)ITEMS;
#pragma unroll 1
                for (uint32_t j = 0; j < end; j++) {
                    const E* e = p + t0 + j;
                    if ((NEIGH && tile == 0 && t0 + j == 0) || test(*e, NEIGH ? e[-1] : *e)) sel |= 1u << j;
                }
            }
            E before = E();
            if constexpr (NEIGH) {
                before = shfl_up_any(x[ITEMS - 1], 1);
                if (lane == 0 && whole) before = p[(int)t0 - 1];
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars.empty[s]);
            if (whole) {
#pragma unroll
                for (int j = 0; j < ITEMS; j++)
                    if (test(x[j], j == 0 ? before : x[j > 0 ? j - 1 : 0])) sel |= 1u << j;
            }
            const uint32_t mine = (uint32_t)__popc(sel);
            const uint32_t c = pipe_lane_sums<32>(mine);
            if (lane == 31) s_wcnt[b][gw] = c;
            pipe_sync(bar, GT);
            const uint32_t wc = lane < (uint32_t)PIPE_COMPUTE ? s_wcnt[b][lane] : 0u;
            const uint32_t wsum = pipe_lane_sums<PIPE_COMPUTE>(wc);
            const uint32_t total = __shfl_sync(0xffffffffu, wsum, PIPE_COMPUTE - 1);
            const uint32_t pos = __shfl_sync(0xffffffffu, wsum - wc, gw) + c - mine;  // selected before this thread's
            const bool lead = gw == PIPE_COMPUTE - 1 && lane == 31;
            if (lead) pipe_put<uint32_t>(st, tile, total, 1u);
            const uint32_t need = PARTITION ? cnt : total;
            uint32_t head = 0;
            if (k > 0) {
                const uint32_t pm = (k - 1u) % PIPE_META;
                if (!mbar_wait_bounded(&bars.agg[pm], ((k - 1u) / PIPE_META) & 1u, st.err))
                    report_error(st.err, TRTC_ERR_LOOKBACK_TIMEOUT);
                head = m_end[(k - 1u) % (2 * PIPE_META)];
            }
            if (k >= (uint32_t)PIPE_META && oldest <= k - PIPE_META) {
                oldest = k - PIPE_META + 1u;
                tail = m_end[(oldest - 1u) % (2 * PIPE_META)];
            }
            if (lead) {
                m_cnt[m] = total;
                m_all[m] = cnt;
                m_start[m] = head % (uint32_t)C;
                m_end[k % (2 * PIPE_META)] = head + need;
                mbar_arrive(&bars.agg[m]);
            }
            for (uint32_t spins = 0; head + need - tail > (uint32_t)C;) {
                if (*(volatile uint32_t*)&m_stored[oldest % (2 * PIPE_META)] == oldest + 1u) {
                    tail = m_end[oldest % (2 * PIPE_META)];
                    oldest++;
                } else if (!spin_continue(spins, st.err)) {
                    report_error(st.err, TRTC_ERR_LOOKBACK_TIMEOUT);
                    break;
                }
            }
            E* r = ring + head % (uint32_t)C + pos;
            E* q = ring + head % (uint32_t)C + total + (t0 - pos);  // rejected, behind the selected ones
#pragma unroll
            for (int j = 0; j < ITEMS; j++) {
                if ((sel >> j) & 1u) *r++ = x[j];
                else if (PARTITION && j < (int)left) *q++ = x[j];
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars.comp[m]);
        }
    } else if (warp < PIPE_COMPUTE * G + PIPE_STORE) {
        // ------------------------------------------------------------ store
        const size_t out_n = out.size();
        for (uint32_t k = warp - PIPE_COMPUTE * G;; k += PIPE_STORE) {
            const uint32_t m = k % PIPE_META;
            if (pipe_store_wait<S, L>(bars, k, &m_last, st.err)) return;
            const uint32_t cnt = m_cnt[m], start = m_start[m];
            const size_t base = m_base[m];
            const size_t lim = base >= out_n ? 0 : out_n - base;
            const uint32_t fit = cnt < lim ? cnt : (uint32_t)lim;
            const E* r = ring + start;
#pragma unroll 8
            for (uint32_t i = lane; i < fit; i += 32) out[base + i] = r[i];
            if constexpr (PARTITION) {
                const size_t fbase = (size_t)m_tile[m] * TILE - base, false_n = out_false.size();
                const uint32_t rej = m_all[m] - cnt;
                const size_t flim = fbase >= false_n ? 0 : false_n - fbase;
                const uint32_t ffit = rej < flim ? rej : (uint32_t)flim;
                const E* f = r + cnt;
#pragma unroll 8
                for (uint32_t i = lane; i < ffit; i += 32) out_false[fbase + i] = f[i];
            }
            __syncwarp();
            if (lane == 0) {
                __threadfence_block();
                *(volatile uint32_t*)&m_stored[k % (2 * PIPE_META)] = k + 1u;
                mbar_arrive(&bars.done[m]);
            }
        }
    } else if (warp == PIPE_COMPUTE * G + PIPE_STORE) {
        // ------------------------------------------------------------ await
        pipe_await_slots(bars.agg, bars.pref, m_tile, st.err, [&](uint32_t m, uint32_t tile) -> bool {
            uint32_t pre = 0;
            if (!pipe_answer<uint32_t>(st, tile, pre)) return false;
            m_base[m] = pre;
            return true;
        });
    } else if (warp == PIPE_COMPUTE * G + PIPE_STORE + 1 && lane == 0) {
        // ------------------------------------------------------------ producer
        const bool aligned = (reinterpret_cast<size_t>(in) & 15u) == 0;
        pipe_produce<G, S, L>(bars, st, tiles, s_first, s_tile, s_bulk, [&](uint32_t s, uint32_t tile, unsigned long long* full) -> bool {
            const size_t base = (size_t)tile * TILE;
            if (!aligned || base + TILE > n) return false;
            const uint32_t lead = NEIGH && base > 0 ? (uint32_t)SM::LEAD : 0u;
            s_bulk[s] = 1u;
            bulk_load_g2s(stage(s) - (int)lead, in + base - lead, (TILE + lead) * (uint32_t)sizeof(E), full);
            return true;
        });
    }
}

// ---------------------------------------------------------------- segmented scan
// Shapes of the segmented scan: 2 groups, tiles of 20 or 10 elements per thread (odd multiples of 16
// bytes, as above), 3 input stages, and slots for 4 tiles of results.
template <class K, class T> struct SpipeShape {
    static constexpr int G = 2, S = 3, R = 4, ITEMS = sizeof(K) + sizeof(T) <= 8 ? 20 : 10;
    static constexpr int TILE = PIPE_COMPUTE * 32 * ITEMS, HALO = 16 / (int)sizeof(K);
    static constexpr size_t KEY_BYTES = (size_t)(TILE + HALO) * sizeof(K);
    static constexpr size_t STAGE = KEY_BYTES + (size_t)TILE * sizeof(T);
    static constexpr size_t SLOTS = S * STAGE;
    static constexpr size_t SMEM = SLOTS + (size_t)R * TILE * sizeof(T);
};

// Scan of the values within segments of equal consecutive keys (EqualTo, Plus; MODE 0 inclusive,
// MODE 1 exclusive behind init) of contiguous arrays.  The tile is scanned on chip without what
// enters it; the store warps add that to the elements before its first head.  What enters a tile is
// the aggregate of the tile before when that holds a head (polled directly), else the prefix CTA's
// answer.  out may be vals itself; it does not overlap the keys.
// st: published words, st2: answers.
template <class K, class T, int MODE>
__global__ void __launch_bounds__(PipeShape<SpipeShape<K, T>::G>::THREADS, 1) scan_by_key_pipe_kernel(const K* keys, const T* vals, T* out,
                                                                                                      size_t n, uint32_t tiles, T init,
                                                                                                      LookbackState st, LookbackState st2) {
    typedef SpipeShape<K, T> SH;
    constexpr int G = SH::G, S = SH::S, R = SH::R, ITEMS = SH::ITEMS;
    constexpr uint32_t TILE = SH::TILE;
    constexpr uint32_t OWN = (1u << ITEMS) - 1u;
    constexpr int VEC = 16 / (int)sizeof(T);
    extern __shared__ __align__(16) unsigned char pipe_smem[];
    constexpr int L = S % G == 0 ? S : S * G;
    __shared__ PipeBars<S, L> bars;
    __shared__ uint32_t s_tile[S], s_bulk[S];
    __shared__ uint32_t m_tile[PIPE_META], m_first[PIPE_META], m_carry_h[PIPE_META];  // (m_first: the tile's first head)
    __shared__ T m_carry[PIPE_META];
    __shared__ T s_wtot[2 * G][PIPE_COMPUTE];
    __shared__ uint32_t s_wfirst[2 * G][PIPE_COMPUTE];  // the warp's first head, TILE when it holds none
    __shared__ uint32_t m_last;
    __shared__ unsigned long long s_first;

    const uint32_t warp = threadIdx.x >> 5, lane = lane_id();
    auto skey = [&](uint32_t s) -> K* { return reinterpret_cast<K*>(pipe_smem + s * SH::STAGE) + SH::HALO; };
    auto sval = [&](uint32_t s) -> T* { return reinterpret_cast<T*>(pipe_smem + s * SH::STAGE + SH::KEY_BYTES); };
    auto slot = [&](uint32_t k) -> T* { return reinterpret_cast<T*>(pipe_smem + SH::SLOTS) + (size_t)(k % R) * TILE; };
    if (threadIdx.x == 0) {
        bars.init(1u);
        m_last = 0xFFFFFFFFu;
        s_first = atomicAdd(st.tile_ctr, 1ull);
    }
    __syncthreads();
    Plus op;
    if (s_first == 0) {
        constexpr int HALF = PipeShape<G>::WARPS / 2;
        // with no other CTA: a tile by this half's warps, whenever all drawn ones are answered (their next
        // ticket is then this tile's) and nobody has drawn for a while; again soon after it
        auto tile_alone = [&](uint32_t tile, const T& carry, bool has) {
            auto* s_chunk = reinterpret_cast<PipeChunk<T, HALF>*>(pipe_smem);
            T* s_x = reinterpret_cast<T*>(pipe_smem + 8192);
            const size_t base = (size_t)tile * TILE;
            const uint32_t cnt = (n - base) < (size_t)TILE ? (uint32_t)(n - base) : TILE;
            PipeRun<T> run;
            for (uint32_t c0 = 0; c0 < cnt; c0 += HALF * 32) {
                const size_t i = base + c0 + threadIdx.x;
                const bool valid = c0 + threadIdx.x < cnt;
                T v = T();
                bool head = false, open;
                if (valid) {
                    v = vals[i];
                    head = i == 0 || !(keys[i] == keys[i - 1]);
                }
                T before = run.v;
                v = pipe_chunk_scan<HALF>(v, head, valid, op, warp, 1u, s_chunk, run, open);
                if constexpr (MODE == 1) {
                    s_x[threadIdx.x] = v;
                    pipe_sync(1u, HALF * 32);
                    if (threadIdx.x > 0) before = s_x[threadIdx.x - 1];
                    pipe_sync(1u, HALF * 32);
                    if (i == base) before = carry;
                    else if (open && has) before = (T)op(carry, before);
                    v = head ? init : (T)op(init, before);
                } else {
                    if (open && has) v = (T)op(carry, v);
                }
                if (valid) out[i] = v;
            }
            if (threadIdx.x == 0) pipe_put<T>(st, tile, run.v, run.open ? 1u : 5u);
        };
        auto draw = [&](uint32_t tile) -> bool {
            const unsigned long long t = (unsigned long long)tile + 1u;
            if (atomicCAS(st.tile_ctr, t, t + 1u) != t) return false;
            if (t == (unsigned long long)tiles + gridDim.x - 1) atomicExch(st.tile_ctr, 0ull);
            return true;
        };
        if (warp < HALF)
            pipe_prefix_scan<T, Plus, true, HALF>(st, st2, tiles, op, nullptr, 0u, 1u,
                                                  PipeSolo<decltype(draw), decltype(tile_alone)>{draw, tile_alone});
        return;
    }
    constexpr uint32_t GT = PIPE_COMPUTE * 32;  // threads of a group

    if (warp < PIPE_COMPUTE * G) {
        // ------------------------------------------------------------ compute
        const uint32_t g = warp / PIPE_COMPUTE, gw = warp % PIPE_COMPUTE, gt = threadIdx.x % GT, bar = 1u + g;
        const uint32_t t0 = gt * ITEMS;
        for (uint32_t k = g;; k += G) {
            const uint32_t s = k % S, m = k % PIPE_META, b = (k / G % 2u) * G + g;
            const bool fail = !mbar_wait_bounded(&bars.full[k % L], (k / L) & 1u, st.err);
            if (fail) report_error(st.err, TRTC_ERR_LOOKBACK_TIMEOUT);
            if (pipe_any(bar, GT, fail)) return;
            const uint32_t tile = s_tile[s];
            if (gt == 0) m_tile[m] = tile;  // (free: tile k - R, later than k - PIPE_META, is waited for below)
            if (tile == PIPE_END) {
                if (gt == 0) {
                    atomicMin(&m_last, k);
                    mbar_arrive(&bars.agg[m]);
                }
                return;
            }
            const size_t base = (size_t)tile * TILE;
            const uint32_t cnt = (n - base) < (size_t)TILE ? (uint32_t)(n - base) : TILE;
            K* kp = skey(s);
            T* vp = sval(s);
            if (!s_bulk[s]) {
                for (uint32_t i = gt; i < cnt; i += GT) {
                    kp[i] = keys[base + i];
                    vp[i] = vals[base + i];
                }
                if (gt == 0 && base > 0) kp[-1] = keys[base - 1];
                smem_proxy_fence();
                pipe_sync(bar, GT);
            }
            K kk[ITEMS];
            T x[ITEMS];
            pipe_load_run<K, ITEMS>(kp + t0, kk);
            pipe_load_run<T, ITEMS>(vp + t0, x);
            K prevk = shfl_up_any(kk[ITEMS - 1], 1);
            if (lane == 0) prevk = kp[(int)t0 - 1];
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars.empty[s]);
            uint32_t hd = 0;  // bit j: element j starts a segment
#pragma unroll
            for (int j = 0; j < ITEMS; j++)
                if (!(kk[j] == (j == 0 ? prevk : kk[j > 0 ? j - 1 : 0]))) hd |= 1u << j;
            if (cnt < TILE) {
                // elements past the end count as heads of value T(); they are not stored
                const uint32_t left = cnt > t0 ? cnt - t0 : 0u;
                if (left < (uint32_t)ITEMS) {
                    hd |= OWN & ~((1u << left) - 1u);
#pragma unroll
                    for (int j = 0; j < ITEMS; j++)
                        if (j >= (int)left) x[j] = T();
                }
            }
            if (tile == 0 && gt == 0) hd |= 1u;
            // running values from the lane's first element or the last head on
#pragma unroll
            for (int j = 1; j < ITEMS; j++)
                if (!((hd >> j) & 1u)) x[j] = (T)op(x[j - 1], x[j]);
            const uint32_t hm = __ballot_sync(0xffffffffu, hd != 0u);
            const uint32_t le = lane == 31u ? 0xffffffffu : ((2u << lane) - 1u);  // lanes <= l
            const uint32_t dist = (hm & le) ? lane - (31u - (uint32_t)__clz(hm & le)) : lane;
            T inc = x[ITEMS - 1];
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const T y = shfl_up_any(inc, d);
                if ((uint32_t)d <= dist) inc = (T)op(y, inc);
            }
            const T ex = shfl_up_any(inc, 1);
            const bool exhd = (hm & (le >> 1)) != 0u;  // a head in lanes < l
            if (lane == 31) s_wtot[b][gw] = inc;
            if (hm == 0u ? lane == 0u : lane == (uint32_t)__ffs(hm) - 1u)
                s_wfirst[b][gw] = hm == 0u ? TILE : t0 + (uint32_t)__ffs(hd) - 1u;
            pipe_sync(bar, GT);
            const uint32_t wf = lane < (uint32_t)PIPE_COMPUTE ? s_wfirst[b][lane] : TILE;
            const uint32_t wall = __ballot_sync(0xffffffffu, wf != TILE);  // warps holding heads
            const uint32_t first = __reduce_min_sync(0xffffffffu, wf);
            const uint32_t whd = wall & ((1u << gw) - 1u);
            T run = T();
            bool run_h = gw > 0u;
            if (gw > 0u) {
                uint32_t w = whd ? 31u - (uint32_t)__clz(whd) : 0u;
                run = s_wtot[b][w];
#pragma unroll 1
                for (w++; w < gw; w++) run = (T)op(run, s_wtot[b][w]);
            }
            if (gw == PIPE_COMPUTE - 1 && lane == 31) {
                const T agg = (!run_h || hm) ? inc : (T)op(run, inc);
                pipe_put<T>(st, tile, agg, wall ? 5u : 1u);
                m_first[m] = first;
                mbar_arrive(&bars.agg[m]);
            }
            if (lane > 0) {
                run = (exhd || !run_h) ? ex : (T)op(run, ex);
                run_h = true;
            }
            // the lane's elements before its first head continue what precedes the lane in the tile
            const uint32_t lf = hd ? (uint32_t)__ffs(hd) - 1u : (uint32_t)ITEMS;
            if (run_h) {
#pragma unroll
                for (int j = 0; j < ITEMS; j++)
                    if (j < (int)lf) x[j] = (T)op(run, x[j]);
            }
            if constexpr (MODE == 1) {
                // the value before each element; before the tile's first head (where what enters the
                // tile comes in as well) bare, behind it with init in front
                T before = run;  // (T() at the tile's first element)
#pragma unroll
                for (int j = 0; j < ITEMS; j++) {
                    const T y = x[j];
                    const bool open = t0 + (uint32_t)j < first;
                    x[j] = ((hd >> j) & 1u) ? init : open ? before : (T)op(init, before);
                    before = y;
                }
            }
            // the slot's last tile is written
            if (k >= (uint32_t)R && !mbar_wait_bounded(&bars.done[(k - R) % PIPE_META], ((k - R) / PIPE_META) & 1u, st.err))
                report_error(st.err, TRTC_ERR_LOOKBACK_TIMEOUT);
            T* r = slot(k) + t0;
            if constexpr (ITEMS * sizeof(T) % 16 == 0) {
                union U { uint4 q[ITEMS * sizeof(T) / 16]; T t[ITEMS]; TRTC_FORCEINLINE U() {} } u;
#pragma unroll
                for (int j = 0; j < ITEMS; j++) u.t[j] = x[j];
#pragma unroll
                for (int j = 0; j < (int)(ITEMS * sizeof(T) / 16); j++) reinterpret_cast<uint4*>(r)[j] = u.q[j];
            } else {
#pragma unroll
                for (int j = 0; j < ITEMS; j++) r[j] = x[j];
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars.comp[m]);
        }
    } else if (warp < PIPE_COMPUTE * G + PIPE_STORE) {
        // ------------------------------------------------------------ store
        const bool aligned = (reinterpret_cast<size_t>(out) & 15u) == 0;
        for (uint32_t k = warp - PIPE_COMPUTE * G;; k += PIPE_STORE) {
            const uint32_t m = k % PIPE_META;
            if (pipe_store_wait<S, L>(bars, k, &m_last, st.err)) return;
            const size_t base = (size_t)m_tile[m] * TILE;
            const uint32_t cnt = (n - base) < (size_t)TILE ? (uint32_t)(n - base) : TILE;
            const bool has = m_carry_h[m] != 0u;
            const uint32_t first = m_first[m] < cnt ? m_first[m] : cnt;
            const T carry = m_carry[m];
            // with what enters the tile (i is before the tile's first head)
            auto entered = [&](uint32_t i, const T& v) -> T {
                if constexpr (MODE == 0) return has ? (T)op(carry, v) : v;
                else return (T)op(init, i == 0 ? carry : has ? (T)op(carry, v) : v);
            };
            const T* r = slot(k);
            if (aligned && cnt == TILE) {
#pragma unroll 4
                for (uint32_t i = lane * VEC; i < TILE; i += 32 * VEC) {
                    union { uint4 q; T t[VEC]; } u;
                    u.q = *reinterpret_cast<const uint4*>(r + i);
                    if (i < first) {
#pragma unroll
                        for (int e = 0; e < VEC; e++)
                            if (i + e < first) u.t[e] = entered(i + e, u.t[e]);
                    }
                    __stcs(reinterpret_cast<uint4*>(out + base + i), u.q);
                }
            } else {
                for (uint32_t i = lane; i < cnt; i += 32) {
                    T v = r[i];
                    if (i < first) v = entered(i, v);
                    out[base + i] = v;
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars.done[m]);
        }
    } else if (warp == PIPE_COMPUTE * G + PIPE_STORE) {
        // ------------------------------------------------------------ await
        pipe_await_slots(bars.agg, bars.pref, m_tile, st.err, [&](uint32_t m, uint32_t tile) -> bool {
            T v = T();
            uint32_t f = 0;
            if (tile > 0) {
                f = pipe_peek<T>(st, tile - 1u, v);
                if (f == 5u) {
                    if constexpr (!LbPack<T>::value) {
                        fence_acq_rel();
                        v = reinterpret_cast<const T*>(st.agg)[tile - 1u];
                    }
                } else {
                    f = pipe_answer<T>(st2, tile, v);
                    if (!f) return false;
                }
            }
            m_carry[m] = v;
            m_carry_h[m] = (f & 4u) ? 1u : 0u;
            return true;
        });
    } else if (warp == PIPE_COMPUTE * G + PIPE_STORE + 1 && lane == 0) {
        // ------------------------------------------------------------ producer
        const bool aligned = ((reinterpret_cast<size_t>(keys) | reinterpret_cast<size_t>(vals)) & 15u) == 0;
        pipe_produce<G, S, L>(bars, st, tiles, s_first, s_tile, s_bulk, [&](uint32_t s, uint32_t tile, unsigned long long* full) -> bool {
            const size_t base = (size_t)tile * TILE;
            if (!aligned || base + TILE > n) return false;
            const uint32_t lead = base > 0 ? (uint32_t)SH::HALO : 0u;
            const uint32_t kb = (TILE + lead) * (uint32_t)sizeof(K), vb = TILE * (uint32_t)sizeof(T);
            s_bulk[s] = 1u;
            mbar_arrive_expect(full, kb + vb);
            bulk_load_g2s_more(skey(s) - (int)lead, keys + base - lead, kb, full);
            bulk_load_g2s_more(sval(s), vals + base, vb, full);
            return true;
        });
    }
}

}  // namespace trtc
