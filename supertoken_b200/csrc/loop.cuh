// The merge loop of one GPU as one persistent cooperative kernel: one CTA per SM takes every step
//     choose the next best pairs -> apply the merges, deltas into the pair table
// without returning to the host; the launch ends when a stop rule fires or the host has maintenance to do.
//
// A late merge changes a few thousand places of a stream of any size, so its cost is the latency of the steps,
// not bandwidth: as four launches per merge (select, worklist, merge, refresh) inside a replayed graph a step
// took 31 us on a 1 MiB corpus and 42-58 us late in a 256 MiB one.  Here the CTAs meet once per merge, at a grid
// barrier when all deltas are in the table: a counter in L2 that every CTA increments (release) and polls
// (acquire), 1.3 us with nothing outstanding.  (Measured on the same 148 CTAs: one CTA collecting flags and
// answering 2.0-2.2 us, all CTAs polling all flags 2.9 us; fewer CTAs are no faster.)  Then every CTA
// re-reads the counts of all candidates, a few hundred slots that are in L2, and takes the same decision from
// the same values.  (With block maxima in shared memory, refreshed through a bitmap of dirty blocks, and a
// vote of the CTAs on the best of them, the same step took 4.3 us instead of 1.5.)
// A second counter keeps the CTAs apart the other way round: a CTA adds its deltas of merge m only when all have
// read the counts that chose merge m (and CTA 0 has reset the step's counters); that wait runs under the rewriting of
// the tiles, but for a delta that finds no place in the CTA's histogram, which waits at once (agg_probe).  Both counters are raised with release and polled with acquire.  (Raised without, `chosen` would rest on
// loads whose values have been used.  The release holds up its warp, so it is done while warp 0 decides: 10 MB of
// mixed text, 3 000 merges, 15.11 ms against 15.08 without any ordering; in front of the ranking, where a CTA barrier waits
// for that warp, 15.30, and with relaxed polls and a fence behind them 16.5.)
//
// A step takes several merges.  Let p1, p2, ... = (a1, b1), (a2, b2), ... be the pairs in selection order (larger count,
// then smaller key), let no ai be a bj with i != j (of a pair of equal tokens no token may occur elsewhere), and let every
// id of the stream be smaller than the new ones.  Then an occurrence of pj overlaps no match of the others, so merging
// them leaves its count as it is.  They make
// only pairs with one of their new tokens; such a pair (x, new i) occurs at most as often as (x, ai) did, and (x, ai),
// which is none of p1 .. pj, came after pj; where the counts are equal the larger key, new > every token of pj,
// loses (and the same for (new i, y) and (bi, y)).  So pj is the best pair after p1 .. pj-1, exactly as if the
// counts had been taken after each merge, and p1 .. pj are applied at once.
// (A new id that the stream holds already may lift a pair that was there: with base_vocab 5 and rows 50 x 012, 50 x 01,
// 60 x 34, 40 x 52 the merge (0,1) -> 5 takes (5,2) from 40 to 90, past (3,4).  Ids at or above base_vocab come from the
// caller: streams with marker ids, merges with ids of their own.  Such merges go one by one until the new ids
// have passed them; the host keeps the bound, LoopArgs::ids_below.)
// The batch ends at the first pair that breaks the rule, at Batch<T>::MAX, and wherever a stop rule or
// maintenance has to be decided first.  On text a batch is 4.7 merges on average (3.9 while no token was to be
// shared at all): the grid barrier, the choice and the flush of the deltas, some 9 of the 12 us of a sparse merge,
// are paid once for all of them.
//
// Nothing else is exchanged: the tiles a merge must visit come out of the pair filter inside each CTA.
//
// All waits are bounded (STBPE_LOOP_WAIT_NS): a CTA that gives up sets STBPE_DERR_TIMEOUT and leaves, and so do
// the others, each at its own limit at the latest.  The cooperative launch guarantees that all CTAs are resident.
#pragma once
#include "kernels.cuh"

struct LoopArgs {
    int target;             // merge count to stop at
    const int2 *forced;     // host-given merges (a, b), applied in order before any choice ...
    int2 one;               // ... or the single one, when forced is null
    int n_forced, forced_new;  // merge i of the launch gets id forced_new + i
    int mode;               // what follows them: LOOP_BEST the best pairs, LOOP_NONE nothing, LOOP_UNTIED the best pairs
                            // while no other pair has the same count
    LoopSync *other_sync;   // counters of the next launch, which this one sets to zero
    i64 filter_count;       // leave to build the pair filter when the merge's count has fallen to this
    int repack_tiles;       // leave for a re-pack at three quarters live from this many tiles on
    int unit_shift;         // tiles per filter unit, log2 (cta_merge)
    i64 grow_keys;          // leave for a larger pair table when a merge could take the number of keys beyond this ...
    int ids_below;          // every id of the stream lies below this (those of the launch's own merges apart)
    const uint32_t *draws;  // LOOP_UNTIED, 16-bit tokens: outputs of the generator that breaks ties; without any, a tie ends the launch
    int n_draws;
};
#define STBPE_DRAWS 1024  // at most

enum { LOOP_BEST, LOOP_NONE, LOOP_UNTIED };

// The arg-max in registers.  With 15-bit ids a pair and its count fit 64 bits whose order is the
// order of the selection (larger count, then smaller key), and a warp's maximum is two redux steps.  That leaves 34
// bits for the count; a stream with more equal pairs is widened before the loop starts.
template <typename T>
struct Best;
template <>
struct Best<uint16_t> {
    typedef u64 type;
    static constexpr i64 COUNTS = 1ll << 34;
    static __device__ __forceinline__ u64 none() { return 0ull; }
    static __device__ __forceinline__ u64 make(u64 key, i64 count) {
        const u64 k30 = ((key >> 32) << 15) | (key & 0x7FFFull);
        return count > 0 ? ((u64)count << 30) | (0x3FFFFFFFull - k30) : 0ull;
    }
    static __device__ __forceinline__ u64 max2(u64 x, u64 y) { return x > y ? x : y; }
    static __device__ __forceinline__ u64 warp_max(u64 v) {
        const uint32_t hi = __reduce_max_sync(0xFFFFFFFFu, (uint32_t)(v >> 32));
        const uint32_t lo = __reduce_max_sync(0xFFFFFFFFu, (uint32_t)(v >> 32) == hi ? (uint32_t)v : 0u);
        return ((u64)hi << 32) | lo;
    }
    static __device__ __forceinline__ Slot slot(u64 v) {
        Slot s;
        s.count = (i64)(v >> 30);
        const u64 k30 = 0x3FFFFFFFull - (v & 0x3FFFFFFFull);
        s.key = v ? ((k30 >> 15) << 32) | (k30 & 0x7FFFull) : STBPE_EMPTY;
        return s;
    }
};
template <>
struct Best<uint32_t> {
    typedef Slot type;
    static __device__ __forceinline__ Slot make(u64 key, i64 count) {
        Slot s;
        s.key = count > 0 ? key : STBPE_EMPTY;
        s.count = count > 0 ? count : 0;
        return s;
    }
    static __device__ __forceinline__ Slot none() { return make(STBPE_EMPTY, 0); }
    static __device__ __forceinline__ Slot max2(const Slot &x, const Slot &y) { return better(y.key, y.count, x.key, x.count) ? y : x; }
    static __device__ __forceinline__ Slot warp_max(Slot v) {
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            Slot o;
            o.key = __shfl_xor_sync(0xFFFFFFFFu, v.key, d);
            o.count = __shfl_xor_sync(0xFFFFFFFFu, v.count, d);
            v = max2(v, o);
        }
        return v;
    }
    static __device__ __forceinline__ Slot slot(const Slot &v) { return v; }
};


// FV: FILTER_ON or FILTER_OFF.  PLANES: 15, or fewer on 16-bit tokens for a launch whose ids, old and new, all stay below
// 2^PLANES - 1; the kernel leaves when the next id would not.  Every tile's 32 x 16 bits per lane are transposed, a quarter of
// the instructions of a dense step and an eighth of a sparse one, and every pair is compared plane by plane.  Nine planes
// and code without the filter took the first 20 merges of 1 GiB from 20.3 to 16.3 ms (24 warps per SM instead of 20: no
// faster); eleven, then thirteen, 8 000 merges of 256 MiB from 121.6 to 118.3 ms.
// DRAW: with the code that breaks ties (16-bit tokens, 15 planes; inside the other kernels it cost 1 % of them, for registers).
template <typename T, int FV, int PLANES, bool DRAW = false>
__global__ void __launch_bounds__(MergeGeom<T>::THREADS, 1) loop_kernel(const __grid_constant__ EngineDev e, const __grid_constant__ LoopArgs la) {
    typedef Best<T> Bs;
    typedef typename Bs::type Bt;
    constexpr int THREADS = MergeGeom<T>::THREADS, WARPS = THREADS / 32;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ int s_ctr[CTR_N];
    constexpr int KB = Batch<T>::MAX, TOP = KB > 1 ? 4 : 1;  // best candidates that each warp hands over
    __shared__ Bt s_sorted[32];           // all warps' best, the first KB in order
    __shared__ Bt s_top[32 * TOP], s_rest[32];  // the warps' best candidates in order; the best of what is left
    __shared__ i64 s_live, s_keys;        // live tokens, keys in the table
    __shared__ i64 s_forced[KB];          // counts of the next host-given pairs
    __shared__ int s_go;                  // merges in this step's batch
    __shared__ int s_tie;                 // this step's merge is drawn among the best pairs
    __shared__ int s_ties, s_drawn, s_used;  // how many they are; which one it is, in ascending order; outputs of the generator used
    __shared__ unsigned int s_err;        // device error bits
    __shared__ int s_ok;                  // every wait so far succeeded
    CtaMerge s;
    unsigned int *s_cand = reinterpret_cast<unsigned int *>(s.carve<T>(smem_raw, s_ctr));  // slots of the candidates
    s.clear();
    DevState *st = e.st;
    LoopSync *sync = e.sync;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned int G = gridDim.x, cta = blockIdx.x;
    int merges_done = st->merges_done, forced_i = 0;
    const int base_vocab = st->base_vocab;
    constexpr bool fv = FV == FILTER_ON;  // (the host launches by DevState::filter_valid)
    MergeCtx mc;
    mc.fv = fv;
    mc.theta.count = st->theta_count, mc.theta.key = st->theta_key;
    unsigned int n_cand = 0;  // candidates this CTA knows
    uint32_t *const s_draws = s_cand + STBPE_CAND_CAP;
    const bool draws = DRAW && la.n_draws > 0;
    if (draws)
        for (int i = tid; i < la.n_draws; i += THREADS) s_draws[i] = la.draws[i];  // (a barrier comes before they are read)
    if (tid == 0) s_ok = 1, s_used = 0;
    auto leave = [&](int why, int stop, const Slot &best, bool valid) {  // one thread of CTA 0
        st->merges_done = merges_done;
        st->run_exit = why;
        st->stopped = stop > 0;
        st->stop_reason = stop;
        st->peek_key = best.key;
        st->peek_count = best.count;
        st->peek_valid = valid;
        st->forced_done = forced_i;
        st->draws_used = DRAW ? s_used : 0;
    };
    WarpStats ws = {0, 0, 0, 0, 0};
    int visited = 0;  // tiles of this CTA in the last step
    if (cta == 0 && tid == 32) {
        if (la.mode != LOOP_BEST) st->n_matches = 0;
        la.other_sync->arrived = la.other_sync->chosen = 0;
    }

#pragma unroll 1
    for (unsigned int step = 0;; ++step) {
        // ---- choose: the counts of all candidates as the last merge left them
        {
            const unsigned int n = __ldcg(&st->n_cand), n_have = min(n, STBPE_CAND_CAP);
            Bt x = Bs::none(), x2 = Bs::none(), rest = Bs::none();  // this thread's best two, and a bound on its others
            auto take = [&](unsigned int at) {
                const Slot y = ldcg_slot(e.table + at);
                const Bt v = Bs::make(y.key, y.count);
                if constexpr (KB > 1) {
                    rest = max(rest, min(v, x2));
                    x2 = max(x2, min(x, v));
                    x = max(x, v);
                } else {
                    x = Bs::max2(x, v);
                }
            };
            // (the place of this thread's first appended candidate is read together with their number)
            unsigned int i_new = n_cand + tid, new_at = i_new < STBPE_CAND_CAP ? __ldcg(e.cand + i_new) : 0u;
#pragma unroll 4
            for (unsigned int i = tid; i < n_cand; i += THREADS) take(s_cand[i]);
#pragma unroll 1
            while (i_new < n_have) {  // appended by the last merges
                s_cand[i_new] = new_at;
                take(new_at);
                i_new += THREADS;
                if (i_new < n_have) new_at = __ldcg(e.cand + i_new);
            }
            n_cand = n_have;
#pragma unroll
            for (int r = 0; r < TOP; ++r) {
                const Bt v = Bs::warp_max(x);
                if (lane == 0) s_top[warp * TOP + r] = v;
                if constexpr (KB > 1) {
                    if (x == v) x = x2, x2 = Bs::none();  // (a pair sits in one slot, so one lane holds it)
                }
            }
            if constexpr (KB > 1) {
                const Bt v = Bs::warp_max(max(x, rest));
                if (lane == 0) s_rest[warp] = v;
                if (tid < 32) s_sorted[tid] = Bs::none();
            }
            if (warp == 0 && lane < KB && forced_i + lane < la.n_forced) {
                const int2 f = la.forced ? la.forced[forced_i + lane] : la.one;
                const i64 at = find_slot(e, ((u64)(uint32_t)f.x << 32) | (uint32_t)f.y);
                s_forced[lane] = at >= 0 ? (i64)__ldcg((const u64 *)&e.table[at].count) : 0;
            }
            if (tid == THREADS - 1) {
                s_live = (i64)__ldcg((const u64 *)&st->n_live);
                s_keys = (i64)__ldcg(&st->n_keys);
                s_err = __ldcg(&st->error) | (n > STBPE_CAND_CAP || __ldcg(&st->cand_state) != STBPE_CAND_READY ? 0x80000000u : 0u);
            }
        }
        __syncthreads();
        if constexpr (KB > 1) {
            // place of this warp's candidates among those of all warps
            constexpr int PER = (WARPS * TOP + 31) / 32;
            Bt v[PER];
#pragma unroll
            for (int r = 0; r < PER; ++r) v[r] = lane + 32 * r < WARPS * TOP ? s_top[lane + 32 * r] : Bs::none();
#pragma unroll 1
            for (int r = 0; r < TOP; ++r) {
                const Bt x = s_top[warp * TOP + r];
                int place = 0;
#pragma unroll
                for (int q = 0; q < PER; ++q) place += __popc(__ballot_sync(0xFFFFFFFFu, v[q] > x));
                if (place > KB) break;  // (one more than a batch holds: the count behind its last member)
                if (lane == 0 && x) s_sorted[place] = x;
            }
            __syncthreads();
        }
        // this CTA has read all that it decides by (if no tie is to be broken, which takes another look)
        if (!draws && tid == THREADS - 1) red_release_u32(&sync->chosen, 1u);
        // warp 0 decides; the lanes of pair j take the j-th best pair (or the j-th one the host gives) and test whether it
        // can be merge j of the batch, given that all before it are
        if (warp == 0) {
            const Bt bound = KB > 1 ? Bs::warp_max(lane < WARPS ? s_rest[lane] : Bs::none()) : Bs::none();
            const Bt mine = KB > 1 ? s_sorted[lane >> 1] : Bs::warp_max(lane < WARPS ? s_top[lane] : Bs::none());
            const bool host = forced_i < la.n_forced;
            const int j = KB > 1 ? lane >> 1 : 0;  // two lanes per pair: one for each of its tokens
            const unsigned int err = s_err;
            const Slot best = Bs::slot(mine);
            const bool dry = (err >> 31) != 0u || !(mc.theta.admits(best.count, best.key) || (best.count <= 0 && mc.theta.count == 0));
            const bool forced = j < KB && forced_i + j < la.n_forced;
            u64 key = best.key;
            i64 count = best.count;
            if (forced) {
                const int2 f = la.forced ? la.forced[forced_i + j] : la.one;
                key = ((u64)(uint32_t)f.x << 32) | (uint32_t)f.y;
                count = s_forced[j];
            }
            const uint32_t a = (uint32_t)(key >> 32), b = (uint32_t)key;
            const uint32_t nw0 = (uint32_t)(la.mode != LOOP_BEST ? la.forced_new + forced_i : base_vocab + merges_done), nw = nw0 + j;
            // a merge drops one token per occurrence of its pair (of a run, all but one), so this many are gone before it
            i64 before = 0;
            if constexpr (KB > 1) {
#pragma unroll
                for (int d = 2; d < 2 * KB; d <<= 1) {
                    const i64 o = __shfl_up_sync(0xFFFFFFFFu, before + count, d);
                    if (lane >= d) before += o;
                }
            }
            const i64 live = s_live - before;
            // every merge makes at most two pairs per match and two per id
            const i64 ids = max((int)nw, la.ids_below), made = min(before + count, ids * (j + 1));
            // a later member: the order is exact so far (which takes new ids above all of the stream), no token is second in
            // one pair and first in another, none is one of the members' new ones (a pair that the host gives, in whatever
            // order, may name one, or be given twice)
            bool out = false;
            if constexpr (KB > 1) {
                const uint32_t same = __match_any_sync(0xFFFFFFFFu, lane >= 2 * KB ? 0x80000000u | lane : lane & 1 ? b : a);
                out = out || (!host && (!(mine > bound) || nw0 < (uint32_t)la.ids_below)) || max(a, b) >= nw0 || (same & ((1u << (lane & ~1)) - 1u) & (lane & 1 ? 0x5555u : 0xAAAAu));
                if (host) {
                    const uint32_t twice = __match_any_sync(0xFFFFFFFFu, lane >= 2 * KB ? 0x80000000u | lane : (a << 15) | b);
                    out = out || (twice & ((1u << (lane & ~1)) - 1u));
                }
            }
            // stop rules of the loop: bpe_trainer.py:4304-4308 (no pairs), :2491-2494 / :4361-4364 (count < 2)
            int stop = 0, why = STBPE_EXIT_STOP;
            bool go = false;
            // LOOP_UNTIED: alone with its count, among the candidates and among the pairs that are not listed.  (The pairs
            // that the merges before it make are rarer than some pair after it, hence rarer than it.)  A slot that is listed
            // twice, as one can be whose pair a merge has lifted again with an id that was there before, takes one place and
            // leaves a gap behind it: then, too, the host looks.
            bool tied = true, draw = false;
            if constexpr (KB > 1) {
                if (la.mode == LOOP_UNTIED) {
                    const Slot after = Bs::slot(max(s_sorted[j + 1], bound));
                    draw = draws && j == 0 && !host && !dry && s_sorted[1] && count == after.count && count > mc.theta.count && count >= 2 &&
                           merges_done < la.target;
                    tied = !s_sorted[j + 1] || count <= after.count || count <= mc.theta.count || count < 2 || merges_done + j >= la.target;
                }
            }
            if (err & 0x7FFFFFFFu) stop = 4;
            else if (la.mode != LOOP_BEST && host && !forced) stop = 0;
            else if (la.mode == LOOP_NONE && !host) stop = 0;
            else if (la.mode == LOOP_UNTIED && !host && !dry && tied && !draw) stop = 0;  // the host looks at what there is
            else if (!host && merges_done + j >= la.target) stop = la.mode == LOOP_BEST ? 1 : 0;
            // maintenance the host does between launches
            else if (!host && dry) why = STBPE_EXIT_REFILL;
            else if (!host && count <= 0) stop = 2;
            else if (!host && count < 2) stop = 3;
            else if (e.n_tiles >= la.repack_tiles && s_live * 4 <= (i64)e.n_tiles * STBPE_TILE * 3) why = STBPE_EXIT_REPACK;
            else if (!fv && e.n_tiles > 0 && count <= la.filter_count) why = STBPE_EXIT_FILTER;
            else if (s_keys + 2 * made + 2 * (j + 1) > la.grow_keys) why = STBPE_EXIT_GROW;
            else if (sizeof(T) == 2 && max(nw, max(a, b)) >= (1u << PLANES) - 1u) why = STBPE_EXIT_WIDEN;
            else go = true;
            draw = __any_sync(0xFFFFFFFFu, draw);
            const uint32_t bad = __ballot_sync(0xFFFFFFFFu, j >= KB || !go || (j > 0 && (out || draw))) | (KB > 1 ? 1u << (2 * KB) : 2u);
            const int nb = lsb(bad) >> (KB > 1 ? 1 : 0);
            if ((KB > 1 ? j < nb && !(lane & 1) : lane < nb) && !draw) {
                s.p->a[j] = a, s.p->b[j] = b, s.p->nw[j] = nw;
                s.p->count[j] = count;
                if (cta == 0) {
                    const int m = merges_done + j;
                    *reinterpret_cast<int2 *>(e.merges + 2 * m) = make_int2((int)a, (int)b);
                    e.merge_counts[m] = count;
                    e.live_before[m] = live;
                    if (j == nb - 1) {
                        st->cur_a = (int)a, st->cur_b = (int)b, st->cur_new = (int)nw;
                        st->cur_count = count;
                    }
                }
            }
            if (lane == 0) {
                s.p->n = nb;
                s.p->chosen = &sync->chosen, s.p->all_chosen = G * (step + 1);
                s_go = nb;
                s_tie = nb > 0 && draw;
                s_ties = 0;
                if (s_tie) s.p->count[0] = count;
                if (cta == 0 && nb == 0) leave(why, stop, best, !dry);
            }
        }
        __syncthreads();
        if constexpr (DRAW) {
            if (s_tie) {
                // The generator picks one of the best pairs in ascending order of their keys (random.Random.randrange: the top
                // bits of an output, again while they are not below the number of pairs).  All CTAs draw the same.
                const i64 c = s.p->count[0];
                u64 *const keys = reinterpret_cast<u64 *>(smem_raw);  // the tiles' slots are free
                for (unsigned int i = tid; i < n_cand; i += THREADS) {
                    const Slot y = ldcg_slot(e.table + s_cand[i]);
                    if (y.count != c) continue;
                    const int at = atoms_add_s32(&s_ties, 1);
                    if (at < STBPE_TIES_CAP) keys[at] = y.key;
                }
                __syncthreads();
                const int n = s_ties;
                constexpr int PER = (STBPE_TIES_CAP + THREADS - 1) / THREADS;
                int place[PER];
                bool odd = n < 2 || n > STBPE_TIES_CAP;  // a pair that is listed twice, or more of them than fit: the host looks
#pragma unroll
                for (int r = 0; r < PER; ++r) {
                    const int i = tid + r * THREADS;
                    place[r] = -1;
                    if (n > STBPE_TIES_CAP || i >= n) continue;
                    const u64 mine = keys[i];
                    int below = 0;
                    for (int q = 0; q < n; ++q) {
                        const u64 other = keys[q];
                        below += other < mine;
                        odd = odd || (other == mine && q != i);
                    }
                    place[r] = below;
                }
                odd = __syncthreads_or(odd);
                if (tid == 0) {
                    int used = s_used, x = -1;
                    if (!odd) {
                        do {
                            x = used < la.n_draws ? (int)(s_draws[used++] >> __clz(n)) : -1;
                        } while (x >= n);
                        if (x >= 0) s_used = used;
                    }
                    s_drawn = x;
                    if (x < 0) {
                        s_go = 0;
                        Slot none;
                        none.key = STBPE_EMPTY, none.count = 0;
                        if (cta == 0) leave(STBPE_EXIT_STOP, 0, none, false);
                    }
                }
                __syncthreads();
#pragma unroll
                for (int r = 0; r < PER; ++r) {
                    if (place[r] < 0 || place[r] != s_drawn) continue;
                    const u64 key = keys[tid + r * THREADS];
                    const int nw = la.forced_new + forced_i;
                    s.p->a[0] = (uint32_t)(key >> 32), s.p->b[0] = (uint32_t)key, s.p->nw[0] = (uint32_t)nw;
                    if (cta == 0) {
                        *reinterpret_cast<int2 *>(e.merges + 2 * merges_done) = make_int2((int)(key >> 32), (int)(uint32_t)key);
                        e.merge_counts[merges_done] = c;
                        e.live_before[merges_done] = s_live;
                        st->cur_a = (int)(key >> 32), st->cur_b = (int)(uint32_t)key, st->cur_new = nw;
                        st->cur_count = c;
                    }
                }
                __syncthreads();
            }
        }
        if (draws && tid == THREADS - 1) red_release_u32(&sync->chosen, 1u);
        const int nb = s_go;
        if (tid < 32 * nb) s.p->set_plane<T>(tid >> 5, lane);  // (barriers of cta_merge come before they are read)
        if (nb == 0 || !s_ok) {
            if (fv && tid == 0 && visited) atomicAdd(&st->n_work, visited);
            add_stats<T>(e, ws);
            return;
        }
        if (cta == 0 && tid == 0 && step == 0) st->n_work = fv ? 0 : -1;  // (what the last step visits is added when the CTAs leave)
        // ---- the merges
        merges_done += nb;
        forced_i += nb;
        mc.m = merges_done;
        mc.zero = cta == G - 1;
        visited = cta_merge<T, false, FV, PLANES>(e, s, mc, la.unit_shift, ws, [&] {
            if (tid == THREADS - 1) {
                BoundedWait wait;
                while (ld_acquire_u32(&sync->chosen) < G * (step + 1))
                    if (!wait.again(st)) {
                        s_ok = 0;
                        break;
                    }
            }
        });
        // ---- grid barrier: every delta is in the table
        if (tid == 0) {
            red_release_u32(&sync->arrived, 1u);
            BoundedWait wait;
            while (ld_acquire_u32(&sync->arrived) < G * (step + 1))
                if (!wait.again(st)) {
                    s_ok = 0;
                    break;
                }
        }
        __syncthreads();
    }
}
