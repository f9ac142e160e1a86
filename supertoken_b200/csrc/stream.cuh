// Token stream: formats, tile loads and the bit-mask view of a tile.
//
// A tile of STBPE_TILE tokens is handled by one warp, 32 consecutive tokens ("a group") per lane.
//   uint16_t stream  one group = 64 bytes = 16 words; word k holds token k in its low and token 16 + k in
//                    its high half.  With that order a compare that leaves one flag bit per half
//                    collects into a 32-bit mask in token order with one shift and one logic operation
//                    per word: acc = (acc >> 1) | flags.
//   uint32_t stream  one group = 128 bytes, tokens in order (ids of 15 bits do not suffice).
// Top bit = first token of a row; all ones = hole (a dropped token, or past the end of the stream).
#pragma once
#include "common.cuh"

template <typename T>
struct Tok;

template <>
struct Tok<uint16_t> {
    static constexpr uint32_t FLAG = 0x8000u, IDMASK = 0x7FFFu, HOLE = 0xFFFFu;
    static constexpr int VEC = 4;     // 16-byte loads per lane and tile
    static constexpr int PITCH = 20;  // shared-memory words per group: 16 + 4, which keeps 16-byte accesses aligned and
                                      // makes the eight lanes of a quarter warp fall on distinct banks
    // token index in memory of stream position p
    static __host__ __device__ __forceinline__ i64 index(i64 p) { return (p & ~(i64)31) + 2 * (p & 15) + ((p >> 4) & 1); }
    static __device__ __forceinline__ int sindex(int p) { return (p >> 5) * 40 + 2 * (p & 15) + ((p >> 4) & 1); }
    // canonical 32-bit form: flag in bit 31, hole / nothing = STBPE_NONE
    static __device__ __forceinline__ uint32_t widen(uint16_t t) {
        const uint32_t w = t;
        return w == HOLE ? STBPE_NONE : ((w & IDMASK) | ((w & FLAG) << 16));
    }
    static __device__ __forceinline__ uint16_t narrow(uint32_t c) {
        return c == STBPE_NONE ? (uint16_t)HOLE : (uint16_t)((c & IDMASK) | ((c >> 16) & FLAG));
    }
    // 16-byte unit j of a group holds tokens 4j .. 4j + 3 and 16 + 4j .. 16 + 4j + 3
    static __device__ __forceinline__ uint32_t unit_mask(int j) { return 0x000F000Fu << (4 * j); }
    // token i (compile-time) of the group whose words are w
    static __device__ __forceinline__ uint32_t get(const uint32_t *w, int i) {
        return widen((uint16_t)(i < 16 ? (w[i] & 0xFFFFu) : (w[i - 16] >> 16)));
    }
};

template <>
struct Tok<uint32_t> {
    static constexpr uint32_t FLAG = STBPE_FLAG, IDMASK = STBPE_IDMASK, HOLE = STBPE_NONE;
    static constexpr int VEC = 8;
    static constexpr int PITCH = 36;
    static __host__ __device__ __forceinline__ i64 index(i64 p) { return p; }
    static __device__ __forceinline__ int sindex(int p) { return (p >> 5) * 36 + (p & 31); }
    static __device__ __forceinline__ uint32_t widen(uint32_t t) { return t; }
    static __device__ __forceinline__ uint32_t narrow(uint32_t c) { return c; }
    static __device__ __forceinline__ uint32_t unit_mask(int j) { return 0xFu << (4 * j); }
    static __device__ __forceinline__ uint32_t get(const uint32_t *w, int i) { return w[i]; }
};

template <typename T>
__device__ __forceinline__ T *tile_ptr(const EngineDev &e, i64 tile) {
    return reinterpret_cast<T *>(e.tiles) + tile * STBPE_TILE;
}

// the tile's 16-byte units, lane-interleaved (coalesced): unit c * 32 + lane into v[c]
template <typename T>
__device__ __forceinline__ void load_units(const EngineDev &e, int tile, int lane, uint4 (&v)[Tok<T>::VEC]) {
    const uint4 *g = reinterpret_cast<const uint4 *>(tile_ptr<T>(e, tile)) + lane;
#pragma unroll
    for (int c = 0; c < Tok<T>::VEC; ++c) v[c] = __ldcg(g + c * 32);
}
// ... and into a warp's shared-memory tile (groups at a pitch of Tok::PITCH words)
template <typename T>
__device__ __forceinline__ void store_units(uint32_t *raw, int lane, const uint4 (&v)[Tok<T>::VEC]) {
#pragma unroll
    for (int c = 0; c < Tok<T>::VEC; ++c) {
        const int u = c * 32 + lane;
        *reinterpret_cast<uint4 *>(raw + (u / Tok<T>::VEC) * Tok<T>::PITCH + (u % Tok<T>::VEC) * 4) = v[c];
    }
}
// this lane's group, straight from memory (kernels that read every token once and never write)
template <typename T>
__device__ __forceinline__ void load_group(const EngineDev &e, int tile, int lane, uint32_t (&w)[Tok<T>::VEC * 4]) {
    const uint4 *g = reinterpret_cast<const uint4 *>(tile_ptr<T>(e, tile)) + lane * Tok<T>::VEC;
#pragma unroll
    for (int j = 0; j < Tok<T>::VEC; ++j) {
        const uint4 q = g[j];
        w[4 * j] = q.x, w[4 * j + 1] = q.y, w[4 * j + 2] = q.z, w[4 * j + 3] = q.w;
    }
}

// One group in registers: L = live tokens, F = tokens that start a row (or holes), eq(id) = tokens with that id.
template <typename T>
struct Group;
// 16-bit stream: the group as 16 bit planes (bit p of plane i = bit i of token p).  The 16 words are two 16 x 16 bit
// matrices side by side; four butterfly steps transpose both at once in 112 instructions, after which the live mask is
// an AND of planes, the row starts are a plane and eq() is one logic operation per plane (15 instead of the 64
// instructions of a compare and a shift per word; a batch of four pairs takes eight of them per group).
struct PlaneId {  // an id as masks: word i = all ones where bit i of the id is set (32-bit stream: word 0 = the id)
    uint4 m[4];
};
template <>
struct Group<uint16_t> {
    uint32_t w[16];
    template <int S>
    __device__ __forceinline__ void exchange(uint32_t mask) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if (i & S) continue;
            const uint32_t x = w[i], y = w[i + S];
            if (S == 8) {
                w[i] = __byte_perm(x, y, 0x6240), w[i + S] = __byte_perm(x, y, 0x7351);
            } else {
                w[i] = (x & mask) | ((y << S) & ~mask);
                w[i + S] = ((x >> S) & mask) | (y & ~mask);
            }
        }
    }
    // PLANES: bits of an id that are looked at; 15, or fewer where every id lies below 2^PLANES - 1 (the planes between
    // them and the last one are then equal to the holes and need not be worked out)
    template <int PLANES>
    __device__ __forceinline__ void load(const uint32_t *group, uint32_t &L, uint32_t &F) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint4 q = *reinterpret_cast<const uint4 *>(group + 4 * j);
            w[4 * j] = q.x, w[4 * j + 1] = q.y, w[4 * j + 2] = q.z, w[4 * j + 3] = q.w;
        }
        exchange<8>(0u);
        exchange<4>(0x0F0F0F0Fu);
        exchange<2>(0x33333333u);
        exchange<1>(0x55555555u);
        uint32_t hole = w[14];
        if (PLANES == 15) {
#pragma unroll
            for (int i = 0; i < 14; i += 2) hole &= w[i] & w[i + 1];  // only a hole has all 15 low bits set
        }
        L = ~hole, F = w[15];
    }
    template <int PLANES>
    __device__ __forceinline__ uint32_t eq(const PlaneId &id) const {
        const uint4 m0 = id.m[0], m1 = id.m[1], m2 = id.m[2], m3 = id.m[3];
        const uint32_t m[15] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w, m2.x, m2.y, m2.z, m2.w, m3.x, m3.y, m3.z};
        uint32_t r = ~(w[0] ^ m[0]);
#pragma unroll
        for (int i = 1; i < PLANES; ++i) r &= ~(w[i] ^ m[i]);
        return r;
    }
};
template <>
struct Group<uint32_t> {
    uint32_t w[32];
    template <int>
    __device__ __forceinline__ void load(const uint32_t *group, uint32_t &L, uint32_t &F) {
        L = F = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint4 q = *reinterpret_cast<const uint4 *>(group + 4 * j);
            w[4 * j] = q.x, w[4 * j + 1] = q.y, w[4 * j + 2] = q.z, w[4 * j + 3] = q.w;
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            if (w[i] != STBPE_NONE) L |= 1u << i;
            if (w[i] & STBPE_FLAG) F |= 1u << i;
            w[i] &= STBPE_IDMASK;
        }
    }
    template <int>
    __device__ __forceinline__ uint32_t eq(const PlaneId &p) const {
        const uint32_t id = p.m[0].x;
        uint32_t m = 0;
#pragma unroll
        for (int i = 0; i < 32; ++i)
            if (w[i] == id) m |= 1u << i;
        return m;
    }
};

// live mask of a group held in registers
template <typename T>
__device__ __forceinline__ uint32_t live_mask(const uint32_t (&w)[Tok<T>::VEC * 4]) {
    uint32_t L = 0;
    if (sizeof(T) == 2) {
        uint32_t nl = 0;
#pragma unroll
        for (int k = 0; k < 16; ++k) nl = (nl >> 1) | (((w[k] & 0x7FFF7FFFu) + 0x00010001u) & 0x80008000u);
        L = ~nl;
    } else {
#pragma unroll
        for (int k = 0; k < Tok<T>::VEC * 4; ++k)
            if (w[k] != STBPE_NONE) L |= 1u << k;
    }
    return L;
}

// Bits q such that q is the next live position above some set position of P inside the word; H = holes.
// S marks the positions right above P.  Where that is a hole it is the lowest of a run of holes, and
// adding it to H carries through the run into the position behind it.
__device__ __forceinline__ uint32_t next_live_bits(uint32_t P, uint32_t H) {
    const uint32_t S = P << 1;
    return (((S & H) + H) & ~H) | (S & ~H);
}

// ... and the previous live positions below the positions of P
__device__ __forceinline__ uint32_t prev_live_bits(uint32_t P, uint32_t H) {
    return __brev(next_live_bits(__brev(P), __brev(H)));
}

// next / previous live position around p in a tile whose live words are bm[0..31], `ne` = words that are
// not zero; STBPE_TILE / -1 when there is none
__device__ __forceinline__ int tile_next(const uint32_t *bm, uint32_t ne, int p) {
    const int w = (p + 1) >> 5;
    if (w > 31) return STBPE_TILE;
    const uint32_t m = bm[w] & (0xFFFFFFFFu << ((p + 1) & 31));
    if (m) return w * 32 + __ffs(m) - 1;
    const uint32_t r = ne & ~((2u << w) - 1u);
    if (!r) return STBPE_TILE;
    const int w2 = __ffs(r) - 1;
    return w2 * 32 + __ffs(bm[w2]) - 1;
}
__device__ __forceinline__ int tile_prev(const uint32_t *bm, uint32_t ne, int p) {
    const int w = p >> 5;
    const uint32_t m = w > 31 ? 0u : bm[w] & ((1u << (p & 31)) - 1u);
    if (m) return w * 32 + 31 - __clz(m);
    const uint32_t r = w > 31 ? ne : ne & ((1u << w) - 1u);
    if (!r) return -1;
    const int w2 = 31 - __clz(r);
    return w2 * 32 + 31 - __clz(bm[w2]);
}

// Calls f(token, next) for every live token of this lane's group, both in canonical form, next = the live
// token that follows (nxt_tile behind the tile's last one).  All lanes call it together.
template <typename T, typename F>
__device__ __forceinline__ void for_each_pair(const uint32_t (&w)[Tok<T>::VEC * 4], uint32_t L, int lane, uint32_t nxt_tile,
                                              F &&f) {
    // first live token of the following lanes
    uint32_t first = STBPE_NONE;
#pragma unroll
    for (int i = 31; i >= 0; --i)
        if ((L >> i) & 1u) first = Tok<T>::get(w, i);
    const uint32_t ne = __ballot_sync(0xFFFFFFFFu, L != 0u);
    const uint32_t above = ne & ~((2u << lane) - 1u);
    const int src = above ? __ffs(above) - 1 : lane;
    const uint32_t other = __shfl_sync(0xFFFFFFFFu, first, src);
    uint32_t next = above ? other : nxt_tile;
#pragma unroll
    for (int i = 31; i >= 0; --i) {
        if ((L >> i) & 1u) {
            const uint32_t t = Tok<T>::get(w, i);
            f(t, next);
            next = t;
        }
    }
}

// ---- dense streams (no merge yet) read as 16-byte units, `THREADS` consecutive units per CTA and step
// v[u] = unit base + u * THREADS + threadIdx.x; nx[u] = first word of the unit behind it (lane 31 only)
template <typename T, int UNROLL, int THREADS>
__device__ __forceinline__ void load_unit_batch(const uint4 *units, i64 base, i64 n_units, uint4 (&v)[UNROLL],
                                                uint32_t (&nx)[UNROLL]) {
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {  // all loads first: several in flight per thread
        const i64 i = base + (i64)u * THREADS + threadIdx.x;
        v[u] = i < n_units ? __ldcs(units + i) : make_uint4(STBPE_NONE, STBPE_NONE, STBPE_NONE, STBPE_NONE);
        nx[u] = ((threadIdx.x & 31) == 31 && i + 1 < n_units) ? __ldcg(reinterpret_cast<const uint32_t *>(units + i + 1)) : STBPE_NONE;
    }
}

// f(t0, t1) for every pair of consecutive tokens that starts in this lane's unit; tokens as stored, top bit
// (Tok::FLAG) = starts a row or lies past the end.  A uint16_t unit is two runs of four tokens (low and
// high halves); the token behind a run sits in the next lane's first word, except at the middle and at the
// end of the group of four lanes.
template <typename T, typename F>
__device__ __forceinline__ void unit_pairs(const uint4 &v, uint32_t nx, F &&f) {
    const int lane = threadIdx.x & 31;
    uint32_t up = __shfl_down_sync(0xFFFFFFFFu, v.x, 1);
    if (lane == 31) up = nx;
    if (sizeof(T) == 2) {
        const uint32_t head = __shfl_sync(0xFFFFFFFFu, v.x, lane & ~3);
        const bool last = (lane & 3) == 3;
        const uint32_t nlo = last ? head >> 16 : up & 0xFFFFu, nhi = last ? up & 0xFFFFu : up >> 16;
        const uint32_t a0 = v.x & 0xFFFFu, a1 = v.y & 0xFFFFu, a2 = v.z & 0xFFFFu, a3 = v.w & 0xFFFFu;
        const uint32_t b0 = v.x >> 16, b1 = v.y >> 16, b2 = v.z >> 16, b3 = v.w >> 16;
        f(a0, a1);
        f(a1, a2);
        f(a2, a3);
        f(a3, nlo);
        f(b0, b1);
        f(b1, b2);
        f(b2, b3);
        f(b3, nhi);
    } else {
        f(v.x, v.y);
        f(v.y, v.z);
        f(v.z, v.w);
        f(v.w, up);
    }
}
