// K3  one merge: find + rewrite + delta counts, by one CTA over its share of the tiles (cta_merge); the
// stand-alone merge_kernel and the persistent loop_kernel both run it.
//
// With M[i] = (id[i]==a && id[j]==b && token j does not start a row), j = the live token behind i,
// evaluated on the pre-merge stream (gpu_tokenizer/utils.py:520-527), token j is dropped when M[i]
// and token i becomes `new` (utils.py:529-531).  The histogram of the result equals a full recount of
// the rewritten rows when these terms are added (the entry of (a,b) itself is zeroed when the merge is
// selected):
//   a != b, per match head (x = the token before it, y = the token behind its partner, both only if in
//   the same row):
//       x exists : if x is the dropped b of a preceding match  +1 (new,new)
//                  else                                         -1 (x,a)  +1 (x,new)
//       y exists : -1 (b,y);  +1 (new,y) unless y heads the next match (whose head then adds
//                  the (new,new) term)
//   a == b, per run of k >= 2 equal tokens (it collapses into ONE new token):
//       head (first token), x exists : -1 (x,a)  +1 (x,new)
//       tail (last token),  y exists : -1 (a,y)  +1 (new,y)
// So the terms of a merge are a histogram of left neighbours x and one of right neighbours y, which the CTA
// collects in shared memory by neighbour id (one 32-bit key per neighbour and side) and turns into
// pair-table adds once per distinct neighbour.
//
// A warp takes a tile through registers into its shared-memory slot (the next tile's loads are in flight
// meanwhile) and works on 32-bit masks, one group of 32 consecutive tokens per lane: live, id a, id b, row
// start.  Match heads, dropped positions and the neighbours' positions all follow from carry arithmetic on
// the masks (next_live_bits) and a few ballots; only neighbours and changed tokens are touched one by one.
// Nothing is compacted: a dropped token becomes a hole and only the 16-byte units that changed are stored.
#pragma once
#include "stream.cuh"

#define STBPE_AGG_BITS 12
#define STBPE_AGG (1 << STBPE_AGG_BITS)   // entries of a CTA's neighbour histogram
#define STBPE_LIST 2048                   // tiles a CTA collects from the pair filter at a time
#define STBPE_LIST_UNITS 64               // filter units (of at most 32 tiles) per batch

template <typename T>
struct MergeGeom {
    static constexpr int WARPS = sizeof(T) == 2 ? 20 : 16;  // one CTA per SM; the wide stream needs twice the shared memory per warp
    static constexpr int THREADS = WARPS * 32;
    static constexpr int RAW_WORDS = 32 * Tok<T>::PITCH;
    static constexpr int WARP_WORDS = RAW_WORDS + 32;  // tile, live masks of the rewritten tile
    static constexpr size_t BYTES = (size_t)WARPS * WARP_WORDS * 4 + (size_t)STBPE_AGG * 10 + STBPE_LIST * 4;
};

enum { CTR_LIST, CTR_AGG, CTR_NN, CTR_BA, CTR_REMOVED, CTR_MATCHES, CTR_SEAM, CTR_FRESH, CTR_TILES, CTR_UNITS, CTR_RECS, CTR_N };

struct CtaMerge {
    uint32_t *warp_mem;    // WARPS x WARP_WORDS
    uint32_t *agg_key;     // neighbour id * 2 + side, or STBPE_NONE
    int *agg_val;
    uint16_t *agg_list;    // taken entries in order of arrival
    uint32_t *list;        // tiles to visit
    int *ctr;              // CTR_N counters

    template <typename T>
    __device__ __forceinline__ unsigned char *carve(unsigned char *base, int *counters) {
        warp_mem = reinterpret_cast<uint32_t *>(base);
        base += (size_t)MergeGeom<T>::WARPS * MergeGeom<T>::WARP_WORDS * 4;
        agg_key = reinterpret_cast<uint32_t *>(base);
        base += STBPE_AGG * 4;
        agg_val = reinterpret_cast<int *>(base);
        base += STBPE_AGG * 4;
        agg_list = reinterpret_cast<uint16_t *>(base);
        base += STBPE_AGG * 2;
        list = reinterpret_cast<uint32_t *>(base);
        base += STBPE_LIST * 4;
        ctr = counters;
        return base;
    }
    __device__ __forceinline__ void clear() const {
        for (int i = threadIdx.x; i < STBPE_AGG; i += blockDim.x) {
            agg_key[i] = STBPE_NONE;
            agg_val[i] = 0;
        }
        if (threadIdx.x < CTR_N) ctr[threadIdx.x] = 0;
    }
};

struct MergeCtx {
    uint32_t a, b, nw;
    int m;         // number of this merge (>= 1)
    bool fv;       // the pair filter is being maintained
    i64 zero;      // this CTA takes this count off the pair (a, b) itself: none survives its own merge.  (Subtracted,
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

// the two pair-table terms of one neighbour: c matches had token `id` on their left (side 0) or right (side 1)
__device__ __forceinline__ u64 gone_key(const MergeCtx &c, uint32_t id, uint32_t side) {
    return side ? (((u64)c.b << 32) | id) : (((u64)id << 32) | c.a);
}
__device__ __forceinline__ u64 made_key(const MergeCtx &c, uint32_t id, uint32_t side) {
    return side ? (((u64)c.nw << 32) | id) : (((u64)id << 32) | c.nw);
}

// Slow path: probe for the entry, claim a free one, or give up.  The entry a key starts at is its low bits:
// while the vocabulary is small (which is when merges have many matches) no two keys share one.
template <bool MG>
static __device__ __noinline__ void agg_probe(uint32_t *agg_key, int *ctr, const EngineDev &e, uint32_t a, uint32_t b, uint32_t nw,
                                              i64 theta_count, u64 theta_key, uint32_t key) {
    // arguments by value: a structure whose address escapes would be re-read from memory after every asm statement
    int *agg_val = reinterpret_cast<int *>(agg_key + STBPE_AGG);
    uint16_t *agg_list = reinterpret_cast<uint16_t *>(agg_val + STBPE_AGG);
    uint32_t h = key & (STBPE_AGG - 1);
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
    MergeCtx c;
    c.a = a, c.b = b, c.nw = nw;
    c.theta.count = theta_count, c.theta.key = theta_key;
    unsigned int fresh = 0;
#pragma unroll 1
    for (int made = 0; made < 2; ++made)
        merge_sink<MG>(e, made ? made_key(c, key >> 1, key & 1u) : gone_key(c, key >> 1, key & 1u), made ? 1 : -1, made != 0, fresh, c.theta);
    if (fresh) atomicAdd(&e.st->n_keys, (u64)fresh);
}

// An entry keeps its key until the histogram is flushed, so a plain load that sees the key is final.
template <bool MG>
__device__ __forceinline__ void agg_add(const CtaMerge &s, const EngineDev &e, const MergeCtx &c, uint32_t id, uint32_t side) {
    const uint32_t key = id * 2u + side, h = key & (STBPE_AGG - 1);
    uint32_t k;
    asm("ld.shared.u32 %0, [%1];" : "=r"(k) : "r"(smem_addr(&s.agg_key[h])));
    if (k == key)
        reds_add_s32(&s.agg_val[h], 1);
    else
        agg_probe<MG>(s.agg_key, s.ctr, e, c.a, c.b, c.nw, c.theta.count, c.theta.key, key);
}

struct WarpStats {  // per lane
    int removed, matches, nn, ba, seam, units, recs;
    int tiles;  // per warp
};

// the records of tiles tile - 1, tile, tile + 1 (two versions each, 192 consecutive bytes), 16 bytes per lane
__device__ __forceinline__ uint4 load_recs3(const EngineDev &e, int tile, int lane) {
    uint4 r = make_uint4(0xFFFFFFFFu, 0u, 0u, 0u);  // version -1, length 0
    const int t = tile - 1 + lane / 4;
    if (lane < 12 && t >= 0 && t < e.n_tiles) r = __ldcg(reinterpret_cast<const uint4 *>(e.recs + 2 * (i64)t) + (lane & 3));
    return r;
}
// lane that holds the first half of the record of tile - 1 + k that is current before merge m
__device__ __forceinline__ int pick_rec(const uint4 &rv, int k, int m) {
    const int v0 = (int)__shfl_sync(0xFFFFFFFFu, rv.x, 4 * k), v1 = (int)__shfl_sync(0xFFFFFFFFu, rv.x, 4 * k + 2);
    const bool ok0 = v0 >= 0 && v0 < m, ok1 = v1 >= 0 && v1 < m;
    return 4 * k + ((ok1 && (!ok0 || v1 > v0)) ? 2 : 0);
}

// One warp, one tile (already in the warp's shared-memory slot; every lane reads and writes its own group of
// 32 tokens only).  `rv`: load_recs3 of the tile.
template <typename T, bool MG>
__device__ __forceinline__ void merge_tile(const EngineDev &e, const CtaMerge &s, const MergeCtx &c, uint32_t *wm, int lane,
                                           int tile, const uint4 &rv, WarpStats &ws) {
    typedef Tok<T> K;
    T *tok = reinterpret_cast<T *>(wm + lane * K::PITCH);
    const bool same = c.a == c.b;

    uint32_t A, B, L, F;
    group_masks((const T *)nullptr, wm + lane * K::PITCH, c.a, c.b, A, B, L, F);
    B &= ~F;  // a partner does not start a row
    const uint32_t ne = __ballot_sync(0xFFFFFFFFu, L != 0u);
    if (ne == 0u) return;  // every token of the tile is gone
    // the live tokens right before and right behind the tile: from the neighbours' records, or by walking
    // when they hold too few tokens
    Halo h;
    const int lp = pick_rec(rv, 0, c.m), ln = pick_rec(rv, 2, c.m);
    const bool near = (int)__shfl_sync(0xFFFFFFFFu, rv.y, lp) >= 2 && (int)__shfl_sync(0xFFFFFFFFu, rv.y, ln) >= 3;
    if (near) {
        h.prev = __shfl_sync(0xFFFFFFFFu, rv.y, lp + 1);
        h.nxt[0] = __shfl_sync(0xFFFFFFFFu, rv.z, ln);
        h.prev_tile = tile - 1;
        h.next_tile = h.next2_tile = tile + 1;
    } else {
        Halo walked;
        gather_halo(e, tile, c.m, walked);
        h = walked;
    }
    const uint32_t H = ~L;
    const uint32_t low = L & (0u - L);                       // this lane's first live token ...
    const uint32_t top = L ? 0x80000000u >> __clz(L) : 0u;   // ... and its last
    const uint32_t above = ne & ~((2u << lane) - 1u), below = ne & ((1u << lane) - 1u);
    const int up = __ffs(above) - 1, down = 31 - __clz(below);  // the next lanes that hold live tokens, if any
    // match heads: positions of A whose next live position is in B
    const uint32_t fb = __ballot_sync(0xFFFFFFFFu, (B & low) != 0u);
    uint32_t M = A & prev_live_bits(B, H);
    if ((A & top) && (above ? ((fb >> up) & 1u) != 0u : h.nxt[0] == c.b)) M |= top;
    // dropped positions: the next live position of every head
    const uint32_t hb = __ballot_sync(0xFFFFFFFFu, (M & top) != 0u);
    const bool carry_in = below == 0u && (B & low) != 0u && (h.prev & STBPE_IDMASK) == c.a;
    uint32_t D = next_live_bits(M, H);
    if (below ? ((hb >> down) & 1u) != 0u : carry_in) D |= low;
    const uint32_t touched = M | D;
    if (__ballot_sync(0xFFFFFFFFu, touched != 0u) == 0u) return;  // nothing to merge here
    ws.matches += __popc(M);
    ws.removed += __popc(D);
    const int first_lane = __ffs(ne) - 1, last_lane = 31 - __clz(ne);
    const bool last_head = ((hb >> last_lane) & 1u) != 0u;  // its partner sits in another tile
    if (!near) {
    } else if (last_head || __any_sync(0xFFFFFFFFu, lane == last_lane && (D & top) && h.nxt[0] == c.a)) {
        h.nxt[1] = __shfl_sync(0xFFFFFFFFu, rv.w, ln);
        h.nxt[2] = __shfl_sync(0xFFFFFFFFu, rv.x, ln + 1);
    }
    if (near && h.prev == c.b) h.prev2 = __shfl_sync(0xFFFFFFFFu, rv.z, lp + 1);

    // ---- the neighbours whose pairs change.  Every left neighbour belongs to one match (a != b) or run (a == b),
    // and so does every right one, so their positions are all that is needed.
    const uint32_t lefts = (same ? M & ~D : M) & ~F;  // heads that have a left neighbour
    const uint32_t ends = same ? D & ~M : D & ~(carry_in ? low : 0u);  // what has its right neighbour accounted for here
    uint32_t X = prev_live_bits(lefts, H), Y = next_live_bits(ends, H);
    const uint32_t xb = __ballot_sync(0xFFFFFFFFu, (lefts & low) != 0u), yb = __ballot_sync(0xFFFFFFFFu, (ends & top) != 0u);
    if (above && ((xb >> up) & 1u)) X |= top;
    if (below && ((yb >> down) & 1u)) Y |= low;
    Y &= ~F;
    int nn = __popc(X & D), ba = __popc(Y & M);  // neighbours that belong to another match: (new, new)
    X &= ~D;
    Y &= ~M;
    uint32_t x_out = STBPE_NONE, y_out = STBPE_NONE;  // neighbours in other tiles
    int y_tile = h.next_tile;
    if (lane == first_lane && (lefts & low)) {
        if (!same && h.prev == c.b && (h.prev2 & STBPE_IDMASK) == c.a)
            nn += 1;
        else
            x_out = h.prev & STBPE_IDMASK;
    }
    if (lane == last_lane) {
        uint32_t y = STBPE_NONE, y2 = STBPE_NONE;
        if (ends & top) {
            y = h.nxt[0], y2 = h.nxt[1];
        } else if (!same && last_head) {
            y = h.nxt[1], y2 = h.nxt[2];
            y_tile = h.next2_tile;
        }
        if (!(y & STBPE_FLAG)) {
            if (!same && y == c.a && y2 == c.b)
                ba += 1;
            else
                y_out = y;
        }
    }
    ws.nn += nn;
    ws.ba += ba;
    if (c.fv && __any_sync(0xFFFFFFFFu, nn + ba != 0) && lane == 0)  // either match of such a pair enters it for its own tile
        filter_set(e, tile, -1, ((u64)c.nw << 32) | c.nw);
#pragma unroll 1
    for (; X; X &= X - 1u) {
        const uint32_t id = tok[K::sindex(__ffs(X) - 1)] & K::IDMASK;
        agg_add<MG>(s, e, c, id, 0u);
        if (c.fv) filter_set(e, tile, -1, made_key(c, id, 0u));
    }
#pragma unroll 1
    for (; Y; Y &= Y - 1u) {
        const uint32_t id = tok[K::sindex(__ffs(Y) - 1)] & K::IDMASK;
        agg_add<MG>(s, e, c, id, 1u);
        if (c.fv) filter_set(e, tile, -1, made_key(c, id, 1u));
    }
    if (x_out != STBPE_NONE || y_out != STBPE_NONE) {
#pragma unroll 1
        for (uint32_t side = 0; side < 2; ++side) {
            const uint32_t id = side ? y_out : x_out;
            if (id == STBPE_NONE) continue;
            agg_add<MG>(s, e, c, id, side);
            if (c.fv) filter_set(e, tile, side ? y_tile : h.prev_tile, made_key(c, id, side));
        }
    }
    // ---- rewrite (no neighbour counted above is a position that changes)
#pragma unroll 1
    for (uint32_t o = M & ~D; o; o &= o - 1u) {
        const int p = __ffs(o) - 1;
        tok[K::sindex(p)] = (T)(c.nw | ((F >> p) & 1u ? K::FLAG : 0u));
    }
#pragma unroll 1
    for (uint32_t o = D; o; o &= o - 1u) tok[K::sindex(__ffs(o) - 1)] = (T)K::HOLE;
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
        if (last_head) {
            ws.seam += 1;
            // a run of a's that goes on in the next tile: the pair that will start at the collapsed token is
            // decided by whoever finds the run's tail, so visit this tile from now on
            if (c.fv && same)
                atomicOr(e.presence + (size_t)((unsigned int)tile >> 5) * STBPE_PPITCH + STBPE_PROWS, 1u << (tile & 31));
        }
    }
    // ---- the record, unless the tile's first three and last two live tokens are as they were
    const uint32_t l2 = L & ~low, l3 = l2 & (l2 - 1u), low3 = L & ~(l3 & (l3 - 1u));
    const uint32_t t2 = L & ~top, top2 = top | (t2 ? 0x80000000u >> __clz(t2) : 0u);
    const bool edge_ok = (lane != first_lane || (l3 && !(touched & low3))) && (lane != last_lane || (t2 && !(touched & top2)));
    if (!__all_sync(0xFFFFFFFFu, edge_ok)) {
        const int lo = pick_rec(rv, 1, c.m);
        // readers of this merge never pick a record stamped m, so payload and stamp need no ordering
        uint32_t *r = reinterpret_cast<uint32_t *>(e.recs + 2 * (i64)tile + ((lo & 2) ? 0 : 1));
        uint32_t *mL = wm + MergeGeom<T>::RAW_WORDS;
        mL[lane] = NL;
        const uint32_t ne2 = __ballot_sync(0xFFFFFFFFu, NL != 0u);
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

// Applies the merge to this CTA's tiles and adds its delta terms to the pair table (or, several ranks, to
// the rank-local delta table).  `unit_shift`: log2 of the tiles per filter unit; CTA c takes the units c,
// c + gridDim.x, ... (words of the filter when there are enough of them, single tiles on a small stream).
// Ends with all of the CTA's adds issued; the caller synchronises.
// `before_adds`: called by every thread between the tiles and the CTA-wide barrier in front of the table adds.
template <typename T, bool MG, typename F>
__device__ __forceinline__ void cta_merge(const EngineDev &e, const CtaMerge &s, const MergeCtx &c, int unit_shift, F &&before_adds) {
    constexpr int WARPS = MergeGeom<T>::WARPS;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t *wm = s.warp_mem + (size_t)warp * MergeGeom<T>::WARP_WORDS;
    WarpStats ws = {0, 0, 0, 0, 0, 0, 0, 0};
    // Without the filter: every tile, consecutive tiles on different CTAs so that a small stream uses all of
    // them.  With it: batches of filter units, each turned into a list of tiles that the warps share.
    unsigned int r1, r2, r3;
    filter_rows(((u64)c.a << 32) | (u64)c.b, r1, r2, r3);
    const i64 n_units = c.fv ? ((i64)e.n_tiles + (1 << unit_shift) - 1) >> unit_shift : blockIdx.x + 1;
    const uint32_t unit_bits = unit_shift == 5 ? 0xFFFFFFFFu : (1u << (1 << unit_shift)) - 1u;
#pragma unroll 1
    for (i64 u0 = blockIdx.x; u0 < n_units; u0 += (i64)STBPE_LIST_UNITS * gridDim.x) {
        int n = (e.n_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;  // tiles blockIdx.x, + gridDim.x, ...
        if (c.fv) {
            const i64 u = u0 + (i64)threadIdx.x * gridDim.x;
            if (threadIdx.x < STBPE_LIST_UNITS && u < n_units) {
                const i64 t0 = u << unit_shift, w = t0 >> 5;
                const unsigned int *g = e.presence + (size_t)w * STBPE_PPITCH;
                uint32_t bits = (__ldcg(g + r1) & __ldcg(g + r2) & __ldcg(g + r3)) | __ldcg(g + STBPE_PROWS);
                bits &= unit_bits << (t0 & 31);
                if (e.n_tiles - w * 32 < 32) bits &= (1u << (e.n_tiles - w * 32)) - 1u;
                if (bits) {
                    int at = atoms_add_s32(&s.ctr[CTR_LIST], __popc(bits));
#pragma unroll 1
                    for (; bits; bits &= bits - 1u) s.list[at++] = (uint32_t)(w * 32 + __ffs(bits) - 1);
                }
            }
            __syncthreads();
            n = s.ctr[CTR_LIST];
        }
        // the loads of a tile are issued before the one before it is worked on
        uint4 v[Tok<T>::VEC], rv;
        int cur = -1;
#pragma unroll 1
        for (int j = warp;; j += WARPS) {
            if (cur >= 0) store_units<T>(wm, lane, v);
            const uint4 rc = rv;
            const int next = j < n ? (c.fv ? (int)s.list[j] : (int)blockIdx.x + j * (int)gridDim.x) : -1;
            if (next >= 0) {
                load_units<T>(e, next, lane, v);
                rv = load_recs3(e, next, lane);
            }
            __syncwarp();
            if (cur >= 0) {
                merge_tile<T, MG>(e, s, c, wm, lane, cur, rc, ws);
                ws.tiles += 1;
                __syncwarp();
            }
            cur = next;
            if (cur < 0) break;
        }
        if (c.fv) {
            __syncthreads();
            if (threadIdx.x == 0) s.ctr[CTR_LIST] = 0;
            if (u0 + (i64)STBPE_LIST_UNITS * gridDim.x < n_units) __syncthreads();
        }
    }
    {
        const int part[8] = {ws.nn, ws.ba, ws.removed, ws.matches, ws.seam, lane == 0 ? ws.tiles : 0, ws.units, ws.recs};
        constexpr int slot[8] = {CTR_NN, CTR_BA, CTR_REMOVED, CTR_MATCHES, CTR_SEAM, CTR_TILES, CTR_UNITS, CTR_RECS};
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int x = __reduce_add_sync(0xFFFFFFFFu, part[k]);
            if (lane == 0 && x) reds_add_s32(&s.ctr[slot[k]], x);
        }
    }
    before_adds();
    __syncthreads();
    // ---- neighbour histogram -> pair table: two lanes per neighbour, one for the pair that is gone and one for
    // the pair that came into being; behind them (new, new), (b, a) and (a, b) itself
    unsigned int fresh = 0;
    const int n = s.ctr[CTR_AGG], total = 2 * n + 3;
#pragma unroll 1
    for (int base = warp * 32; base < total; base += WARPS * 32) {
        const int i = base + lane;
        const bool made = i < 2 * n ? (i & 1) != 0 : i == 2 * n;
        u64 key = 0;
        i64 delta = 0;
        int h = -1;
        if (i < 2 * n) {
            h = s.agg_list[i >> 1];
            const uint32_t k = s.agg_key[h];
            delta = s.agg_val[h];
            key = made ? made_key(c, k >> 1, k & 1u) : gone_key(c, k >> 1, k & 1u);
        } else if (i == 2 * n) {
            key = ((u64)c.nw << 32) | c.nw;
            delta = s.ctr[CTR_NN];
        } else if (i == 2 * n + 1) {
            key = ((u64)c.b << 32) | c.a;
            delta = s.ctr[CTR_BA];
        } else if (i == 2 * n + 2) {
            key = ((u64)c.a << 32) | c.b;
            delta = c.zero;
        }
        __syncwarp();  // both lanes of the entry have read it
        if (h >= 0 && !made) {
            s.agg_key[h] = STBPE_NONE;
            s.agg_val[h] = 0;
        }
        if (delta) merge_sink<MG>(e, key, made ? delta : -delta, made, fresh, c.theta);
    }
    fresh = __reduce_add_sync(0xFFFFFFFFu, fresh);
    if (lane == 0 && fresh) reds_add_s32(&s.ctr[CTR_FRESH], (int)fresh);
    __syncthreads();
    DevState *st = e.st;
    if (threadIdx.x < CTR_N) {
        const int k = threadIdx.x, x = s.ctr[k];
        s.ctr[k] = 0;
        if (x) {  // results unused: reductions
            if (k == CTR_REMOVED) atomicAdd((u64 *)&st->n_live, (u64)(-(i64)x));
            if (k == CTR_MATCHES) atomicAdd((u64 *)&st->n_matches, (u64)x);
            if (k == CTR_SEAM) atomicAdd(&st->n_fixups, (unsigned int)x);
            if (k == CTR_FRESH && !MG) atomicAdd(&st->n_keys, (u64)x);
            if (k == CTR_TILES) {
                if (c.fv) atomicAdd(&st->n_work, x);
                atomicAdd(&st->tile_bytes_in, (u64)x * (STBPE_TILE * sizeof(T) + 2 * sizeof(TileRec)));
            }
            if (k == CTR_UNITS) atomicAdd(&st->tile_bytes_out, (u64)x * 16);
            if (k == CTR_RECS) atomicAdd(&st->tile_bytes_out, (u64)x * sizeof(TileRec));
        }
    }
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
    c.a = (uint32_t)st->cur_a, c.b = (uint32_t)st->cur_b, c.nw = (uint32_t)st->cur_new;
    c.m = st->merges_done;
    c.fv = st->filter_valid != 0;
    c.zero = 0;  // done when the merge was selected
    c.theta.count = st->theta_count, c.theta.key = st->theta_key;
    if (!c.fv && blockIdx.x == 0 && threadIdx.x == 0) st->n_work = -1;
    __syncthreads();
    cta_merge<T, MG>(e, s, c, unit_shift, [] {});
}
