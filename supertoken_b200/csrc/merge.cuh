// K3  a batch of merges: find + rewrite + delta counts, by one CTA over its share of the tiles (cta_merge); the
// stand-alone merge_kernel (always one merge) and the persistent loop_kernel both run it.
//
// With M[i] = (id[i]==a && id[j]==b && token j does not start a row), j = the live token behind i,
// evaluated on the pre-merge stream (gpu_tokenizer/utils.py:520-527), token j is dropped when M[i]
// and token i becomes `new` (utils.py:529-531).  A run of k >= 2 equal tokens (a == b) collapses into ONE new
// token.  In a batch no pair's second token is another's first, so no position belongs to two matches and
// applying the merges together leaves the stream that applying them one after the other leaves (loop.cuh
// says when the next best pairs may form a batch).
//
// The histogram of the result equals a full recount of the rewritten rows when these terms are added (the entries
// of the merged pairs themselves are zeroed when the merges are selected).  For every match (run) of pair k,
// x = the token before its head and y = the token behind its last token, both only if in the same row:
//       x exists : if x is the dropped token of a match of pair i   -1 (b_i,a_k)  +1 (new_i,new_k)
//                  else                                              -1 (x,a_k)    +1 (x,new_k)
//       y exists : if y heads a match: nothing, that match has x    else  -1 (b_k,y)  +1 (new_k,y)
// So the terms are a histogram of left neighbours x and one of right neighbours y per pair, which the CTA
// collects in shared memory by neighbour id (one 32-bit key per neighbour, pair and side) and turns into
// pair-table adds once per distinct neighbour, and a small matrix of matches that touch.
//
// A warp takes a tile through registers into its shared-memory slot (the next tile's loads are in flight
// meanwhile) and works on 32-bit masks, one group of 32 consecutive tokens per lane: live, row start and, per
// pair, id a and id b.  Match heads and dropped positions follow from carry arithmetic on the masks
// (next_live_bits) and a few ballots; only neighbours and changed tokens are touched one by one.
// Nothing is compacted: a dropped token becomes a hole and only the 16-byte units that changed are stored.
#pragma once
#include "stream.cuh"

#define STBPE_AGG_BITS 12
#define STBPE_AGG (1 << STBPE_AGG_BITS)   // entries of a CTA's neighbour histogram
#define STBPE_LIST 2048                   // tiles a CTA collects from the pair filter at a time
#define STBPE_LIST_UNITS 256              // filter units (of at most 8 tiles) per batch
static_assert(STBPE_LIST_UNITS * 8 <= STBPE_LIST, "a batch of units fits the list");

// Pairs of a batch.  Late in a run on text 5.6 of the next best pairs on average can go together when eight may (3.6 of
// four, 6.7 of twelve), and what a late merge costs is latency.  (Twelve: 6 % less per late merge of 256 MiB, 3 % more
// per early one of 1 GiB, where the fourth bit of the pair number costs registers in every tile.)  The wide stream, whose ids leave
// the neighbour histogram's keys no room for a pair number, takes one at a time.
template <typename T>
struct Batch;
template <>
struct Batch<uint16_t> {
    static constexpr int MAX = 8;
    // neighbour key: 15-bit id, side, pair
    static __device__ __forceinline__ uint32_t key(uint32_t id, uint32_t side, uint32_t k) { return id | (side << 15) | (k << 16); }
    static __device__ __forceinline__ uint32_t id(uint32_t key) { return key & 0x7FFFu; }
    static __device__ __forceinline__ uint32_t side(uint32_t key) { return (key >> 15) & 1u; }
    static __device__ __forceinline__ uint32_t pair(uint32_t key) { return key >> 16; }
    // entry the probe starts at: while the vocabulary is small (which is when merges have many matches) the neighbours
    // of one pair fall on distinct entries, and the pairs of a batch start far apart
    static __device__ __forceinline__ uint32_t home(uint32_t key) { return key * 2u + side(key) + pair(key) * 1171u; }
};
template <>
struct Batch<uint32_t> {
    static constexpr int MAX = 1;
    static __device__ __forceinline__ uint32_t key(uint32_t id, uint32_t side, uint32_t) { return id * 2u + side; }
    static __device__ __forceinline__ uint32_t id(uint32_t key) { return key >> 1; }
    static __device__ __forceinline__ uint32_t side(uint32_t key) { return key & 1u; }
    static __device__ __forceinline__ uint32_t pair(uint32_t) { return 0u; }
    static __device__ __forceinline__ uint32_t home(uint32_t key) { return key; }
};
#define STBPE_LOOP_WAIT_NS 4000000000ull
__device__ __forceinline__ u64 loop_timer_ns() {
    u64 t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void red_release_u32(unsigned int *p, unsigned int v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned int ld_acquire_u32(const unsigned int *p) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// retries of a bounded wait; false when the time is up or another wait has given up
struct BoundedWait {
    u64 t0;
    unsigned int n;
    __device__ __forceinline__ BoundedWait() : t0(0), n(0) {}
    __device__ __forceinline__ bool again(DevState *st) {
        if ((++n & 1023u) != 0u) return true;
        const u64 t = loop_timer_ns();
        if (t0 == 0) t0 = t;
        if (t - t0 > STBPE_LOOP_WAIT_NS) atomicOr(&st->error, STBPE_DERR_TIMEOUT);
        return (*(volatile unsigned int *)&st->error & STBPE_DERR_TIMEOUT) == 0u;
    }
};

struct BatchPairs {  // in shared memory
    PlaneId pa[8], pb[8];  // a and b once more, as Group::eq takes them
    uint32_t a[8], b[8], nw[8];
    i64 count[8];
    int touch[64];  // matches of pair i (row) followed at once by one of pair k (column)
    int n;
    // the pair table stays as it is until this counter has reached this value: all CTAs have then read what they choose the
    // batch by (null: they read nothing while the batch is applied)
    const unsigned int *chosen;
    unsigned int all_chosen;
    // called by the 32 lanes of a warp: word i of the masks is all ones where bit i of the id is set
    template <typename T>
    __device__ __forceinline__ void set_plane(int k, int lane) {
        const uint32_t id = lane < 16 ? a[k] : b[k];
        reinterpret_cast<uint32_t *>(pa)[(lane & 16 ? (int)sizeof(pa) / 4 : 0) + k * 16 + (lane & 15)] =
            sizeof(T) == 4 ? id : 0u - ((id >> (lane & 15)) & 1u);
    }
};

template <typename T>
struct MergeGeom {
    static constexpr int WARPS = sizeof(T) == 2 ? 20 : 16;  // one CTA per SM; the wide stream needs twice the shared memory per warp
    static constexpr int THREADS = WARPS * 32;
    static constexpr int RAW_WORDS = 32 * Tok<T>::PITCH;
    static constexpr int WARP_WORDS = RAW_WORDS + 32 * 8 + STBPE_TILE / 2;  // tile, masks of its groups, places of heads and ends
    static constexpr size_t BYTES = (size_t)WARPS * WARP_WORDS * 4 + (size_t)STBPE_AGG * 10 + STBPE_LIST * 5 + STBPE_LIST_UNITS * Batch<T>::MAX + sizeof(BatchPairs);
};

enum { CTR_LIST, CTR_NEXT, CTR_AGG, CTR_REMOVED, CTR_FRESH, CTR_N };

struct CtaMerge {
    uint32_t *warp_mem;    // WARPS x WARP_WORDS
    BatchPairs *p;
    uint32_t *agg_key;     // Batch<T>::key, or STBPE_NONE
    int *agg_val;
    uint16_t *agg_list;    // taken entries in order of arrival
    uint32_t *list;        // tiles to visit ...
    unsigned char *list_pairs;  // ... and the pairs that may occur there
    unsigned char *unit_bits;  // [pair][unit] tiles of the filter units at hand
    int *ctr;              // CTR_N counters

    template <typename T>
    __device__ __forceinline__ unsigned char *carve(unsigned char *base, int *counters) {
        warp_mem = reinterpret_cast<uint32_t *>(base);
        base += (size_t)MergeGeom<T>::WARPS * MergeGeom<T>::WARP_WORDS * 4;
        p = reinterpret_cast<BatchPairs *>(base);
        base += sizeof(BatchPairs);
        agg_key = reinterpret_cast<uint32_t *>(base);
        base += STBPE_AGG * 4;
        agg_val = reinterpret_cast<int *>(base);
        base += STBPE_AGG * 4;
        agg_list = reinterpret_cast<uint16_t *>(base);
        base += STBPE_AGG * 2;
        list = reinterpret_cast<uint32_t *>(base);
        base += STBPE_LIST * 4;
        list_pairs = base;
        base += STBPE_LIST;
        unit_bits = base;
        base += STBPE_LIST_UNITS * Batch<T>::MAX;
        ctr = counters;
        return base;
    }
    __device__ __forceinline__ void clear() const {
        for (int i = threadIdx.x; i < STBPE_AGG; i += blockDim.x) {
            agg_key[i] = STBPE_NONE;
            agg_val[i] = 0;
        }
        if (threadIdx.x < CTR_N) ctr[threadIdx.x] = 0;
        if (threadIdx.x < 64) p->touch[threadIdx.x] = 0;
    }
};

// How a kernel knows whether the pair filter is being maintained: compiled for streams without it, with it, or for both.
enum { FILTER_OFF, FILTER_ON, FILTER_ASK };

struct MergeCtx {
    int m;         // number of the batch's last merge (>= 1)
    bool fv;       // the pair filter is being maintained
    bool zero;     // this CTA takes the counts off the pairs (a, b) themselves: none survives its own merge.  (Subtracted,
                   // not overwritten: an id the host gives may already occur, and its pairs are being added to.)
    Theta theta;   // threshold of the candidate list (one rank)
};

// a delta of the merge, into the pair table (one rank) or the rank-local delta table
template <bool MG>
__device__ __forceinline__ void merge_sink(const EngineDev &e, u64 key, i64 delta, bool made, unsigned int &fresh, const Theta &theta) {
    if (MG)
        ltable_add(e, key, delta);
    else
        table_add<NOTE_CAND>(e, key, delta, made, fresh, theta);
}

// shared-memory atomics through the .shared state space (generic ones are far slower on this part)
__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ int atoms_add_s32(int *p, int v) {
    int old;
    asm volatile("atom.shared.add.s32 %0, [%1], %2;" : "=r"(old) : "r"(smem_addr(p)), "r"(v) : "memory");
    return old;
}
__device__ __forceinline__ uint32_t atoms_cas_u32(uint32_t *p, uint32_t cmp, uint32_t val) {
    uint32_t old;
    asm volatile("atom.shared.cas.b32 %0, [%1], %2, %3;" : "=r"(old) : "r"(smem_addr(p)), "r"(cmp), "r"(val) : "memory");
    return old;
}
__device__ __forceinline__ uint32_t lds_u32_volatile(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(v) : "r"(smem_addr(p)) : "memory");
    return v;
}

// the two pair-table terms of one neighbour: matches of pair k had token `id` on their left (side 0) or right (side 1)
__device__ __forceinline__ u64 gone_key(const BatchPairs *p, uint32_t k, uint32_t id, uint32_t side) {
    return side ? (((u64)p->b[k] << 32) | id) : (((u64)id << 32) | p->a[k]);
}
__device__ __forceinline__ u64 made_key(const BatchPairs *p, uint32_t k, uint32_t id, uint32_t side) {
    return side ? (((u64)p->nw[k] << 32) | id) : (((u64)id << 32) | p->nw[k]);
}

// Slow path: probe for the entry, claim a free one, or give up and add to the pair table, in the middle of the tiles: other
// CTAs may still be choosing the batch by its counts.
template <typename T, bool MG>
static __device__ __noinline__ void agg_probe(uint32_t *agg_key, int *ctr, const EngineDev &e, const BatchPairs *p, i64 theta_count, u64 theta_key,
                                              uint32_t key) {
    // arguments by value: a structure whose address escapes would be re-read from memory after every asm statement
    typedef Batch<T> B;
    int *agg_val = reinterpret_cast<int *>(agg_key + STBPE_AGG);
    uint16_t *agg_list = reinterpret_cast<uint16_t *>(agg_val + STBPE_AGG);
    uint32_t h = B::home(key) & (STBPE_AGG - 1);
#pragma unroll 1
    for (int probe = 0; probe < 16; ++probe) {
        uint32_t k = lds_u32_volatile(&agg_key[h]);
        if (k == STBPE_NONE) {
            k = atoms_cas_u32(&agg_key[h], STBPE_NONE, key);
            if (k == STBPE_NONE) {
                agg_list[atoms_add_s32(&ctr[CTR_AGG], 1)] = (uint16_t)h;
                k = key;
            }
        }
        if (k == key) {
            reds_add_s32(&agg_val[h], 1);
            return;
        }
        h = (h + 1) & (STBPE_AGG - 1);
    }
    if (!MG && p->chosen) {
        BoundedWait wait;
        while (ld_acquire_u32(p->chosen) < p->all_chosen)
            if (!wait.again(e.st)) return;  // the launch ends with STBPE_DERR_TIMEOUT
    }
    Theta theta;
    theta.count = theta_count, theta.key = theta_key;
    unsigned int fresh = 0;
#pragma unroll 1
    for (int made = 0; made < 2; ++made)
        merge_sink<MG>(e, made ? made_key(p, B::pair(key), B::id(key), B::side(key)) : gone_key(p, B::pair(key), B::id(key), B::side(key)), made ? 1 : -1,
                       made != 0, fresh, theta);
    if (fresh) atomicAdd(&e.st->n_keys, (u64)fresh);
}

// An entry keeps its key until the histogram is flushed, so a plain load that sees the key is final.
template <typename T, bool MG>
__device__ __forceinline__ void agg_add(const CtaMerge &s, const EngineDev &e, const MergeCtx &c, uint32_t key) {
    const uint32_t h = Batch<T>::home(key) & (STBPE_AGG - 1);
    uint32_t k;
    asm("ld.shared.u32 %0, [%1];" : "=r"(k) : "r"(smem_addr(&s.agg_key[h])));
    if (k == key)
        reds_add_s32(&s.agg_val[h], 1);
    else
        agg_probe<T, MG>(s.agg_key, s.ctr, e, s.p, c.theta.count, c.theta.key, key);
}

// two at once (STBPE_NONE: no neighbour): the look-ups overlap, and the lanes that have to probe for either do it together
template <typename T, bool MG>
__device__ __forceinline__ void agg_add2(const CtaMerge &s, const EngineDev &e, const MergeCtx &c, uint32_t key0, uint32_t key1) {
    const uint32_t h0 = Batch<T>::home(key0) & (STBPE_AGG - 1), h1 = Batch<T>::home(key1) & (STBPE_AGG - 1);
    uint32_t x0, x1;
    asm("ld.shared.u32 %0, [%1];" : "=r"(x0) : "r"(smem_addr(&s.agg_key[h0])));
    asm("ld.shared.u32 %0, [%1];" : "=r"(x1) : "r"(smem_addr(&s.agg_key[h1])));
    if (key0 != STBPE_NONE && x0 == key0) {
        reds_add_s32(&s.agg_val[h0], 1);
        key0 = STBPE_NONE;
    }
    if (key1 != STBPE_NONE && x1 == key1) {
        reds_add_s32(&s.agg_val[h1], 1);
        key1 = STBPE_NONE;
    }
#pragma unroll 1
    while (key0 != STBPE_NONE || key1 != STBPE_NONE) {
        if (key0 == STBPE_NONE) key0 = key1, key1 = STBPE_NONE;
        agg_probe<T, MG>(s.agg_key, s.ctr, e, s.p, c.theta.count, c.theta.key, key0);
        key0 = STBPE_NONE;
    }
}

// the pair (x, y) of the batch, or n when there is none (a token that starts a row, or nothing, has more bits than an id)
__device__ __forceinline__ int find_pair(const BatchPairs *p, uint32_t x, uint32_t y) {
    int k = 0;
#pragma unroll 1
    while (k < p->n && (p->a[k] != x || p->b[k] != y)) ++k;
    return k;
}

struct WarpStats {  // per lane, over all steps of a launch but for `removed`
    int removed, seam, units, recs;
    i64 tiles;  // of the CTA
};
// Statistics of a launch into the device state.  Called by the whole CTA at its end.
template <typename T>
__device__ __forceinline__ void add_stats(const EngineDev &e, const WarpStats &ws) {
    __shared__ u64 sums[3];
    if (threadIdx.x < 3) sums[threadIdx.x] = 0;
    __syncthreads();
    const unsigned int part[3] = {(unsigned int)ws.seam, (unsigned int)ws.units, (unsigned int)ws.recs};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const u64 lo = __reduce_add_sync(0xFFFFFFFFu, part[k] & 0xFFFFu), hi = __reduce_add_sync(0xFFFFFFFFu, part[k] >> 16);
        if ((threadIdx.x & 31) == 0 && (lo | hi)) atomicAdd(&sums[k], lo + (hi << 16));
    }
    __syncthreads();
    DevState *st = e.st;
    if (threadIdx.x == 0) {
        if (sums[0]) atomicAdd(&st->n_fixups, (unsigned int)sums[0]);
        if (ws.tiles) atomicAdd(&st->tile_bytes_in, (u64)ws.tiles * (STBPE_TILE * sizeof(T) + 2 * sizeof(TileRec)));
        if (sums[1] | sums[2]) atomicAdd(&st->tile_bytes_out, sums[1] * 16 + sums[2] * sizeof(TileRec));
    }
}

// the records of tiles tile - 1, tile, tile + 1 (two versions each, 192 consecutive bytes), 16 bytes per lane
__device__ __forceinline__ uint4 load_recs3(const EngineDev &e, int tile, int lane) {
    uint4 r = make_uint4(0xFFFFFFFFu, 0u, 0u, 0u);  // version -1, length 0
    const int t = tile - 1 + lane / 4;
    if (lane < 12 && t >= 0 && t < e.n_tiles) r = __ldcg(reinterpret_cast<const uint4 *>(e.recs + 2 * (i64)t) + (lane & 3));
    return r;
}
// Which version of each record is current before merge m: bit 4k + 2 of the result is set when it is the second one of
// tile - 1 + k (its first half sits in lane 4k + 2, else in lane 4k).
__device__ __forceinline__ uint32_t pick_recs(const uint4 &rv, int m) {
    const int own = (int)rv.x, other = (int)__shfl_xor_sync(0xFFFFFFFFu, rv.x, 2);
    const bool ok = own >= 0 && own < m, ok_other = other >= 0 && other < m;
    return __ballot_sync(0xFFFFFFFFu, ok && (!ok_other || own > other));
}
// index of the lowest set bit.  (One find-leading-one; __ffs is a bit reversal on top of it, and both run at an eighth of
// the rate of ordinary instructions.)
__device__ __forceinline__ int lsb(uint32_t x) { return 31 - __clz(x & (0u - x)); }

template <int S>
struct SideTag {
    static constexpr int value = S;
};

// One warp, one tile (already in the warp's shared-memory slot; every lane reads and writes its own group of
// 32 tokens only).  `rv`: load_recs3 of the tile; `pm`: the pairs that may occur in it (bit k = pair k).
template <typename T, bool MG, int FV, int PLANES>
__device__ __forceinline__ void merge_tile(const EngineDev &e, const CtaMerge &s, const MergeCtx &c, uint32_t *wm, int lane,
                                           int tile, uint32_t pm, const uint4 &rv, WarpStats &ws) {
    typedef Tok<T> K;
    constexpr bool MANY = Batch<T>::MAX > 1;
    const bool fv = FV == FILTER_ASK ? c.fv : FV == FILTER_ON;
    T *tok = reinterpret_cast<T *>(wm + lane * K::PITCH);
    const BatchPairs *const P = s.p;

    uint32_t L, F;
    Group<T> grp;
    grp.template load<PLANES>(wm + lane * K::PITCH, L, F);
    const uint32_t ne = __ballot_sync(0xFFFFFFFFu, L != 0u);
    if (ne == 0u) return;  // every token of the tile is gone
    const uint32_t H = ~L;
    const uint32_t low = L & (0u - L);                       // this lane's first live token ...
    const uint32_t top = L ? 0x80000000u >> __clz(L) : 0u;   // ... and its last
    const uint32_t above = ne & ~((2u << lane) - 1u), below = ne & ((1u << lane) - 1u);
    const int up = lsb(above), down = 31 - __clz(below);  // the next lanes that hold live tokens, if any
    // The live tokens right before and right behind the tile: from the neighbours' records, or by walking when they hold
    // too few tokens.  A sparse visit reads them when it turns out to need them; in a dense one most tiles do, and the
    // shuffles run beside the comparisons (first 20 merges of 1 GiB 16.5 ms, 17.4 where they are read late).
    Halo h;
    uint32_t second = 0;  // pick_recs of the tile
    auto read_halo = [&] {
        second = pick_recs(rv, c.m);
        const int lp = second & 4u ? 2 : 0, ln = second & 0x400u ? 10 : 8;
        const uint32_t enough = __ballot_sync(0xFFFFFFFFu, (int)rv.y >= (lane < 4 ? 2 : 3));
        if ((enough >> lp) & (enough >> ln) & 1u) {
            h.prev = __shfl_sync(0xFFFFFFFFu, rv.y, lp + 1);
            h.prev2 = __shfl_sync(0xFFFFFFFFu, rv.z, lp + 1);
            h.nxt[0] = __shfl_sync(0xFFFFFFFFu, rv.z, ln);
            h.nxt[1] = __shfl_sync(0xFFFFFFFFu, rv.w, ln);
            h.nxt[2] = __shfl_sync(0xFFFFFFFFu, rv.x, ln + 1);
            h.prev_tile = tile - 1;
            h.next_tile = h.next2_tile = tile + 1;
        } else {
            Halo walked;
            gather_halo(e, tile, c.m, walked);
            h = walked;
        }
    };
    if (FV != FILTER_ON) read_halo();
    // Dropped tokens: positions of some b_k whose previous live position holds a_k.  k0, k1, k2: bits of k there.
    uint32_t D = 0, k0 = 0, k1 = 0, k2 = 0;
    uint32_t firsts = 0, seconds = 0;  // pairs whose a is this lane's last token, whose b is its first
#pragma unroll 1
    for (uint32_t left = pm; left; left &= left - 1u) {
        const int k = MANY ? lsb(left) : 0;
        const uint32_t A = grp.template eq<PLANES>(P->pa[k]), B = grp.template eq<PLANES>(P->pb[k]) & ~F;  // a partner does not start a row
        const uint32_t d = next_live_bits(A, H) & B;
        D |= d;
        if (A & top) firsts |= 1u << k;
        if (B & low) seconds |= 1u << k;
        if (MANY) {
            if (k & 1) k0 |= d;
            if (k & 2) k1 |= d;
            if (k & 4) k2 |= d;
        }
    }
    // heads: the previous live position of every dropped one
    uint32_t M = prev_live_bits(D, H);
    // matches across lanes: kt = pair of the one that this lane's last token heads, kl = of the one whose partner is its
    // first, -1 for none
    auto drop_first = [&](int k) {
        D |= low;
        if (MANY) {
            if (k & 1) k0 |= low;
            if (k & 2) k1 |= low;
            if (k & 4) k2 |= low;
        }
    };
    int kt = -1, kl = -1;
    {
        const uint32_t both = firsts & __shfl_sync(0xFFFFFFFFu, seconds, above ? up : lane);
        if (above && both) kt = lsb(both), M |= top;
        kl = __shfl_sync(0xFFFFFFFFu, kt, below ? down : lane);
        if (!below) kl = -1;
        if (L != 0u && kl >= 0) drop_first(kl);
    }
    // ---- the tile's edges: what stands beyond them matters, and the tile's record changes, only when one of the first
    // three or last two live tokens is touched or could belong to a match with the tile next to it
    const int first_lane = lsb(ne), last_lane = 31 - __clz(ne);
    const uint32_t l2 = L & ~low, l3 = l2 & (l2 - 1u), low3 = L & ~(l3 & (l3 - 1u));
    const uint32_t t2 = L & ~top, top2 = top | (t2 ? 0x80000000u >> __clz(t2) : 0u);
    const bool edge = (lane == first_lane && (!l3 || ((M | D) & low3) || seconds)) || (lane == last_lane && (!t2 || ((M | D) & top2) || firsts));
    const bool edges = __any_sync(0xFFFFFFFFu, edge);
    bool last_head = false;  // the last token's partner sits in another tile
    bool carry_in = false;   // this lane's first token is the partner of a token in another tile
    if (edges) {
        if (FV == FILTER_ON) read_halo();
        if (lane == last_lane) {
            uint32_t both = 0;
            for (uint32_t o = firsts; o; o &= o - 1u)
                if (h.nxt[0] == P->b[lsb(o)]) both = o & (0u - o);
            if (both) kt = lsb(both), M |= top;
        }
        if (lane == first_lane) {
            for (uint32_t o = seconds; o; o &= o - 1u)
                if ((h.prev & STBPE_IDMASK) == P->a[lsb(o)]) kl = lsb(o);
            if (kl >= 0) carry_in = true, drop_first(kl);
        }
        last_head = (__ballot_sync(0xFFFFFFFFu, kt >= 0) >> last_lane) & 1u;
    }
    const uint32_t touched = M | D;
    if (__ballot_sync(0xFFFFFFFFu, touched != 0u) == 0u) return;  // nothing to merge here
    ws.removed += __popc(D);
    const uint32_t heads = M & ~D;  // (a position in both is inside a run of equal tokens)
    const uint32_t ends = D & ~M;   // last tokens of matches and runs
    // of a match whose head sits in the tile before, the head's tile takes care (of a run, the last token's tile)
    const uint32_t own = ends & ~(carry_in && P->a[kl] != P->b[kl] ? low : 0u);
    // ---- the neighbours whose pairs change.  Heads (left neighbours) and own ends (right neighbours) go through a list
    // and are taken 32 at a time, one per lane, whatever group they sit in and whichever of the two they are.  What a
    // lane has to know of another's group it reads from shared memory.  Tokens that are read as neighbours are never
    // rewritten: in front of a head stands no head, a dropped token counts by its pair, and a head behind an end is skipped.
    // (A visit has 2.4 matches on average over the 8 000 merges of a 256 MiB corpus, mostly in lanes of their own: a lane that
    // takes its head and then its end holds up the warp for both.  Every lane walking
    // over its own matches waited for the fullest lane: first 20 merges of 1 GiB 23.9 ms instead of 20.3.)
    uint4 *const sa = reinterpret_cast<uint4 *>(wm + MergeGeom<T>::RAW_WORDS), *const sb = sa + 32;
    T *const all = reinterpret_cast<T *>(wm);
    sa[lane] = make_uint4(L, D, k0, k1);
    sb[lane] = make_uint4(k2, F, heads, (uint32_t)kt);
    uint16_t *const list = reinterpret_cast<uint16_t *>(sb + 32);
    uint32_t at, sum;  // places in front of this lane's, places in all: heads, and ends in the upper half
    {
        if (__any_sync(0xFFFFFFFFu, ((heads & (heads - 1u)) | (own & (own - 1u))) != 0u)) {  // some lane has several
            const uint32_t n = (uint32_t)__popc(heads) | ((uint32_t)__popc(own) << 16);
            at = n;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t o = __shfl_up_sync(0xFFFFFFFFu, at, d);
                if (lane >= d) at += o;
            }
            sum = __shfl_sync(0xFFFFFFFFu, at, 31);
            at -= n;
        } else {
            const uint32_t hb = __ballot_sync(0xFFFFFFFFu, heads != 0u), eb = __ballot_sync(0xFFFFFFFFu, own != 0u), lt = (1u << lane) - 1u;
            at = (uint32_t)__popc(hb & lt) | ((uint32_t)__popc(eb & lt) << 16);
            sum = (uint32_t)__popc(hb) | ((uint32_t)__popc(eb) << 16);
        }
        uint16_t *lh = list + (at & 0xFFFFu), *le = list + (sum & 0xFFFFu) + (at >> 16);
        uint32_t oh = heads, oe = own;
#pragma unroll 1
        while (oh | oe) {
            if (oh) {
                const int q = 31 - __clz(oh);
                oh ^= 1u << q;
                *lh++ = (uint16_t)(lane * 32 + q);
            }
            if (oe) {
                const int r = 31 - __clz(oe);
                oe ^= 1u << r;
                *le++ = (uint16_t)(STBPE_TILE + lane * 32 + r);
            }
        }
    }
    __syncwarp();
    auto pair_at = [&](const uint4 &x, uint32_t x2, int r) {
        return MANY ? (int)(((x.z >> r) & 1u) | (((x.w >> r) & 1u) << 1) | (((x2 >> r) & 1u) << 2)) : 0;
    };
    // One entry of the list: rewrites the token and returns its neighbour's key.  SIDE: 0 a head, 1 an end, 2 either.
    auto visit = [&](int item, auto side) -> uint32_t {
        constexpr int SIDE = decltype(side)::value;
        const int at = item & (STBPE_TILE - 1), l = at >> 5, q = at & 31;
        const bool end = SIDE == 2 ? item >= STBPE_TILE : SIDE == 1;
        uint4 x = sa[l], y = sb[l];
        const uint32_t over = x.x & ~((2u << q) - 1u), under = x.x & ((1u << q) - 1u);
        const int k = !MANY ? 0 : end || over ? pair_at(x, y.x, end ? q : lsb(over)) : (int)y.w;
        const uint32_t nw = P->nw[k];
        const bool starts = !end && ((y.y >> q) & 1u);  // first of its row: no left neighbour
        all[K::sindex(at)] = (T)(end ? K::HOLE : nw | (starts ? K::FLAG : 0u));
        if (starts) return STBPE_NONE;
        uint32_t n = end ? over : under;
        int ln = l;
        if (!n) {
            const uint32_t lanes = end ? ne & ~((2u << l) - 1u) : ne & ((1u << l) - 1u);
            if (lanes) {
                ln = end ? lsb(lanes) : 31 - __clz(lanes);
                x = sa[ln], y = sb[ln];
                n = x.x;
            }
        }
        uint32_t id;
        int i = -1, tile2 = -1;  // pair of the match that ends in front of this one; tile of the neighbour, if another
        if (n) {
            const int p = end ? lsb(n) : 31 - __clz(n);
            id = (uint32_t)all[K::sindex(ln * 32 + p)] & K::IDMASK;
            if (((end ? y.y | y.z : x.y) >> p) & 1u) {
                if (end) return STBPE_NONE;  // another row, or the head of a match, which counts the pair
                i = pair_at(x, y.x, p);
            }
        } else if (end) {
            id = h.nxt[0];
            if ((id & STBPE_FLAG) || find_pair(P, id, h.nxt[1]) < P->n) return STBPE_NONE;
            tile2 = h.next_tile;
        } else {
            id = h.prev & STBPE_IDMASK;
            const int j = find_pair(P, h.prev2 & STBPE_IDMASK, h.prev);
            if (j < P->n) i = j;
            tile2 = h.prev_tile;
        }
        if (fv) filter_set(e, tile, tile2, made_key(P, (uint32_t)k, i >= 0 ? P->nw[i] : id, end));
        if (i < 0) return Batch<T>::key(id, end, (uint32_t)k);
        reds_add_s32(&s.p->touch[i * 8 + k], 1);
        return STBPE_NONE;
    };
    // Many matches in the tile: a head and an end per lane and round, each by code of its own, which is less of it (first 20
    // merges of 1 GiB 16.42 ms, 16.7 if each takes one side of either kind); with the filter, hardly any tile has as many.
    const int n_heads = (int)(sum & 0xFFFFu), n_ends = (int)(sum >> 16);
    if (FV != FILTER_ON && n_heads + n_ends > 32) {
#pragma unroll 1
        for (int base = lane; base - lane < max(n_heads, n_ends); base += 32) {
            uint32_t head = STBPE_NONE, end = STBPE_NONE;
            if (base < n_heads) head = visit((int)list[base], SideTag<0>());
            if (base < n_ends) end = visit((int)list[n_heads + base], SideTag<1>());
            agg_add2<T, MG>(s, e, c, head, end);
        }
    } else {
#pragma unroll 1
        for (int base = lane; base - lane < n_heads + n_ends; base += 32)
            if (base < n_heads + n_ends) {
                const uint32_t key = visit((int)list[base], SideTag<2>());
                if (key != STBPE_NONE) agg_add<T, MG>(s, e, c, key);
            }
    }
    // dropped tokens that are no end of this tile's: inside a run, or of a match that starts in the tile before
#pragma unroll 1
    for (uint32_t o = D & ~own; o;) {
        const int r = 31 - __clz(o);
        o ^= 1u << r;
        tok[K::sindex(r)] = (T)K::HOLE;
    }
    __syncwarp();
    if (last_head && lane == last_lane) {
        if (P->a[kt] != P->b[kt]) {
            const uint32_t y = h.nxt[1];
            const int i = find_pair(P, y, h.nxt[2]);
            if (i < P->n) {
                // y's tile counts the two touching matches, but sees the dropped token only, not the new one here
                if (fv) filter_set(e, tile, -1, ((u64)P->nw[kt] << 32) | P->nw[i]);
            } else if (!(y & STBPE_FLAG)) {
                agg_add<T, MG>(s, e, c, Batch<T>::key(y, 1u, (uint32_t)kt));
                if (fv) filter_set(e, tile, h.next2_tile, made_key(P, kt, y, 1u));
            }
        } else if (fv) {
            // a run of a's that goes on in the next tile: the pair that will start at the collapsed token is
            // decided by whoever finds the run's tail, so visit this tile from now on
            atomicOr(e.presence + (size_t)((unsigned int)tile >> 5) * STBPE_PPITCH + STBPE_PROWS, 1u << (tile & 31));
        }
    }
    // ---- what changed goes back
    {
        uint4 *g = reinterpret_cast<uint4 *>(tile_ptr<T>(e, tile)) + lane * K::VEC;
#pragma unroll
        for (int j = 0; j < K::VEC; ++j)
            if (touched & K::unit_mask(j)) {
                g[j] = *reinterpret_cast<const uint4 *>(wm + lane * K::PITCH + 4 * j);
                ws.units += 1;
            }
    }
    const uint32_t NL = L & ~D;
    const int newlen = __reduce_add_sync(0xFFFFFFFFu, __popc(NL));
    if (lane == 0) {
        e.tile_live[tile] = (unsigned int)newlen;
        if (last_head) ws.seam += 1;
    }
    // ---- the record, unless the tile's first three and last two live tokens are as they were
    if (edges) {
        // readers of this merge never pick a record stamped m, so payload and stamp need no ordering
        uint32_t *r = reinterpret_cast<uint32_t *>(e.recs + 2 * (i64)tile + ((second & 0x40u) ? 0 : 1));
        const uint32_t ne2 = __ballot_sync(0xFFFFFFFFu, NL != 0u), n2 = NL & (NL - 1u), n3 = n2 & (n2 - 1u);
        const uint32_t two = __ballot_sync(0xFFFFFFFFu, n2 != 0u), three = __ballot_sync(0xFFFFFFFFu, n3 != 0u);
        const int fl = lsb(ne2), ll = 31 - __clz(ne2);
        if (ne2 && ((three >> fl) & (two >> ll) & 1u)) {  // the usual case: one lane holds the first three, one the last two
            if (lane == fl) {
                ws.recs += 1;
                r[0] = (uint32_t)c.m;
                r[1] = (uint32_t)newlen;
                r[2] = K::widen(tok[K::sindex(lsb(NL))]);
                r[3] = K::widen(tok[K::sindex(lsb(n2))]);
                r[4] = K::widen(tok[K::sindex(lsb(n3))]);
            }
            if (lane == ll) {
                const int p = 31 - __clz(NL);
                r[5] = K::widen(tok[K::sindex(p)]);
                r[6] = K::widen(tok[K::sindex(31 - __clz(NL ^ (1u << p)))]);
            }
            return;
        }
        uint32_t *mL = wm + MergeGeom<T>::RAW_WORDS;
        mL[lane] = NL;
        __syncwarp();
        if (lane == 0) {
            ws.recs += 1;
            r[0] = (uint32_t)c.m;
            r[1] = (uint32_t)newlen;
            const T *all = reinterpret_cast<const T *>(wm);
            int p = -1;
#pragma unroll 1
            for (int i = 0; i < 5; ++i) {  // first three live tokens, then the last two backwards
                if (i == 3) p = STBPE_TILE;
                uint32_t t = STBPE_NONE;
                if (i < 3 ? i < newlen : i - 3 < newlen) {
                    p = i < 3 ? tile_next(mL, ne2, p) : tile_prev(mL, ne2, p);
                    t = K::widen(all[K::sindex(p)]);
                }
                r[2 + i] = t;
            }
        }
    }
}

// Applies the batch of merges to this CTA's tiles and adds its delta terms to the pair table (or, several ranks, to
// the rank-local delta table).  `unit_shift`: log2 of the tiles per filter unit; CTA c takes the units c,
// c + gridDim.x, ... (words of the filter when there are enough of them, single tiles on a small stream).
// Returns the tiles it visited.  Ends behind a CTA-wide barrier with all of the CTA's adds issued, the last ones by thread 0.
// `before_adds`: called by every thread between the tiles and the CTA-wide barrier in front of the table adds.
template <typename T, bool MG, int FV, int PLANES, typename F>
__device__ __forceinline__ int cta_merge(const EngineDev &e, const CtaMerge &s, const MergeCtx &c, int unit_shift, WarpStats &ws, F &&before_adds) {
    constexpr int WARPS = MergeGeom<T>::WARPS;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t *wm = s.warp_mem + (size_t)warp * MergeGeom<T>::WARP_WORDS;
    ws.removed = 0;
    int visited = 0;
    const bool fv = FV == FILTER_ASK ? c.fv : FV == FILTER_ON;
    const int nb = Batch<T>::MAX > 1 ? s.p->n : 1;
    if (!fv) __syncthreads();  // the pairs are in place (with the filter, the barriers of the list come first)
    // Without the filter: every tile, consecutive tiles on different CTAs so that a small stream uses all of
    // them.  With it: batches of filter units, each turned into a list of tiles that the warps share.
    const i64 n_units = fv ? ((i64)e.n_tiles + (1 << unit_shift) - 1) >> unit_shift : blockIdx.x + 1;
    const uint32_t unit_bits = (1u << (1 << unit_shift)) - 1u;
#pragma unroll 1
    for (i64 u0 = blockIdx.x; u0 < n_units; u0 += (i64)STBPE_LIST_UNITS * gridDim.x) {
        int n = (e.n_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;  // tiles blockIdx.x, + gridDim.x, ...
        if (fv) {
            if (u0 != blockIdx.x) {  // the list before this one has been worked off
                __syncthreads();
                if (threadIdx.x == 0) s.ctr[CTR_LIST] = s.ctr[CTR_NEXT] = 0;
                __syncthreads();
            }
            // one thread per pair and unit asks the filter ...
            int lg = 2;
            while (lg < 8 && u0 + ((i64)gridDim.x << lg) < n_units) ++lg;
#pragma unroll 2
            for (int it = threadIdx.x; it < nb << lg; it += WARPS * 32) {
                const int k = it >> lg;
                const i64 u = u0 + (i64)(it & ((1 << lg) - 1)) * gridDim.x, t0 = u << unit_shift;
                uint32_t bits = 0;
                if (u < n_units) {
                    const unsigned int *g = e.presence + (size_t)(t0 >> 5) * STBPE_PPITCH;
                    unsigned int r1, r2, r3;
                    filter_rows(((u64)s.p->a[k] << 32) | (u64)s.p->b[k], r1, r2, r3);
                    bits = (__ldcg(g + r1) & __ldcg(g + r2) & __ldcg(g + r3)) | __ldcg(g + STBPE_PROWS);
                    bits = (bits >> (t0 & 31)) & unit_bits;
                    if (e.n_tiles - t0 < 8) bits &= (1u << (e.n_tiles - t0)) - 1u;
                }
                s.unit_bits[it] = (unsigned char)bits;
            }
            __syncthreads();
            // ... and a warp per four units lists the tiles that any pair needs: lane = tile lane % 8 of unit lane / 8
#pragma unroll 1
            for (int i = warp; i < 1 << (lg - 2); i += WARPS) {
                const uint32_t own = lane < nb ? reinterpret_cast<const uint32_t *>(s.unit_bits)[(lane << (lg - 2)) + i] : 0u;
                const uint32_t any = __reduce_or_sync(0xFFFFFFFFu, own);
                if (any == 0u) continue;
                uint32_t pairs = 0;
#pragma unroll 1
                for (int q = 0; q < nb; ++q) pairs |= ((__shfl_sync(0xFFFFFFFFu, own, q) >> lane) & 1u) << q;
                int at0 = 0;
                if (lane == 0) at0 = atoms_add_s32(&s.ctr[CTR_LIST], __popc(any));
                at0 = __shfl_sync(0xFFFFFFFFu, at0, 0) + __popc(any & ((1u << lane) - 1u));
                if (pairs) {
                    s.list[at0] = (uint32_t)((u0 + (i64)(4 * i + (lane >> 3)) * gridDim.x) << unit_shift) + (lane & 7);
                    s.list_pairs[at0] = (unsigned char)pairs;
                }
            }
            __syncthreads();
            n = s.ctr[CTR_LIST];
        }
        visited += n;
        // the loads of a tile are issued before the one before it is worked on; of a list, a warp takes the
        // next tile that is left (visiting every tile, the warps stay together: fixed shares save an atomic per tile)
        // (Loading the first tile of a step under the table adds of the one before, where every tile is visited: no faster on a
        // small stream, and 8 % slower on 1 GiB, for the registers.)
        uint4 v[Tok<T>::VEC], rv;
        int next = -1, taken = 0;
        uint32_t next_pairs = (1u << nb) - 1u;
        auto fetch = [&](int j) {
            next = j < n ? (fv ? (int)s.list[j] : (int)blockIdx.x + j * (int)gridDim.x) : -1;
            if (next < 0) return;
            if (fv) next_pairs = s.list_pairs[j];
            load_units<T>(e, next, lane, v);
            rv = load_recs3(e, next, lane);
            if (fv && lane == 0) taken = atoms_add_s32(&s.ctr[CTR_NEXT], 1);
        };
        fetch(warp);
#pragma unroll 1
        for (int j = warp; next >= 0;) {
            const int tile = next;
            const uint32_t pairs = next_pairs;
            const uint4 rc = rv;
            store_units<T>(wm, lane, v);
            j = fv ? __shfl_sync(0xFFFFFFFFu, taken, 0) + WARPS : j + WARPS;
            fetch(j);
            __syncwarp();
            merge_tile<T, MG, FV, PLANES>(e, s, c, wm, lane, tile, pairs, rc, ws);
            __syncwarp();
        }
    }
    ws.tiles += visited;
    const int removed = __reduce_add_sync(0xFFFFFFFFu, ws.removed);
    if (lane == 0 && removed) reds_add_s32(&s.ctr[CTR_REMOVED], removed);
    before_adds();
    __syncthreads();
    DevState *st = e.st;
    if (threadIdx.x == MergeGeom<T>::THREADS - 1) {
        s.ctr[CTR_LIST] = s.ctr[CTR_NEXT] = 0;
        const int x = s.ctr[CTR_REMOVED];
        s.ctr[CTR_REMOVED] = 0;
        if (x) {  // one dropped token per match; results unused: reductions
            atomicAdd((u64 *)&st->n_live, (u64)(-(i64)x));
            atomicAdd((u64 *)&st->n_matches, (u64)x);
        }
    }
    // ---- neighbour histogram -> pair table: two lanes per neighbour, one for the pair that is gone and one for
    // the pair that came into being; behind them, likewise, the matches that touch, and the merged pairs themselves
    constexpr int KB = Batch<T>::MAX, TOUCH = 2 * KB * 8;
    unsigned int fresh = 0;
    const int n = s.ctr[CTR_AGG], total = 2 * n + TOUCH + KB;
#pragma unroll 1
    for (int base = warp * 32; base < total; base += WARPS * 32) {
        const int i = base + lane, t = i - 2 * n;
        bool made = (i & 1) != 0;
        u64 key = 0;
        i64 delta = 0;
        int *used = nullptr;
        if (t < 0) {
            const int h = s.agg_list[i >> 1];
            const uint32_t x = s.agg_key[h], k = Batch<T>::pair(x), id = Batch<T>::id(x), side = Batch<T>::side(x);
            used = &s.agg_val[h];
            delta = *used;
            key = made ? made_key(s.p, k, id, side) : gone_key(s.p, k, id, side);
        } else if (t < TOUCH) {
            used = &s.p->touch[t >> 1];
            delta = *used;
            const int l = t >> 4, r = (t >> 1) & 7;
            if (delta) key = made ? ((u64)s.p->nw[l] << 32) | s.p->nw[r] : ((u64)s.p->b[l] << 32) | s.p->a[r];
        } else {
            made = false;
            if (c.zero && t - TOUCH < nb) {
                key = ((u64)s.p->a[t - TOUCH] << 32) | s.p->b[t - TOUCH];
                delta = s.p->count[t - TOUCH];
            }
        }
        __syncwarp();  // both lanes of the entry have read it
        if (used && !made) {
            if (t < 0) s.agg_key[used - s.agg_val] = STBPE_NONE;
            *used = 0;
        }
        if (delta) merge_sink<MG>(e, key, made ? delta : -delta, made, fresh, c.theta);
    }
    fresh = __reduce_add_sync(0xFFFFFFFFu, fresh);
    if (lane == 0 && fresh) reds_add_s32(&s.ctr[CTR_FRESH], (int)fresh);
    __syncthreads();
    if (threadIdx.x == 0) {
        const int x = s.ctr[CTR_FRESH];
        s.ctr[CTR_FRESH] = s.ctr[CTR_AGG] = 0;
        if (x && !MG) atomicAdd(&st->n_keys, (u64)x);
    }
    return visited;
}

// One merge as a launch of its own (several ranks, timed runs): the merge that DevState names.
template <typename T, bool MG>
__global__ void __launch_bounds__(MergeGeom<T>::THREADS, 1) merge_kernel(const __grid_constant__ EngineDev e, int unit_shift) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ int s_ctr[CTR_N];
    DevState *st = e.st;
    if (st->stopped || st->exchange_only || st->merges_done < 1) return;
    CtaMerge s;
    s.carve<T>(smem_raw, s_ctr);
    s.clear();
    MergeCtx c;
    if (threadIdx.x == 0) s.p->n = 1, s.p->a[0] = (uint32_t)st->cur_a, s.p->b[0] = (uint32_t)st->cur_b, s.p->nw[0] = (uint32_t)st->cur_new, s.p->chosen = nullptr;
    c.m = st->merges_done;
    c.fv = st->filter_valid != 0;
    c.zero = false;  // done when the merge was selected
    c.theta.count = st->theta_count, c.theta.key = st->theta_key;
    if (!c.fv && blockIdx.x == 0 && threadIdx.x == 0) st->n_work = -1;
    __syncthreads();
    if (threadIdx.x < 32) s.p->set_plane<T>(0, (int)threadIdx.x);
    WarpStats ws = {0, 0, 0, 0, 0};
    const int visited = cta_merge<T, MG, FILTER_ASK, 15>(e, s, c, unit_shift, ws, [] {});
    if (c.fv && threadIdx.x == 0 && visited) atomicAdd(&st->n_work, visited);
    add_stats<T>(e, ws);
}
