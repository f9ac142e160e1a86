// Kernels of the BPE merge-loop engine (sm_100a).  See common.cuh for the data layout.
#pragma once
#include "merge.cuh"

// ---------------------------------------------------------------------------------------
// K1  pack: bytes / ids -> stream tokens, row-start flags, tile records
// ---------------------------------------------------------------------------------------
// identity byte -> id map of the reference's packer (gpu_tokenizer/cpu_packer.py:17-26).
// Streaming copy, one group of 32 tokens per thread: 32 source bytes become the group's 16 words (a byte
// permutation per word).  `at` = stream position of src[0]; groups that the append covers only in part, and
// sources that are not 16-byte aligned relative to the groups, are written token by token.
template <typename T>
__device__ __forceinline__ void put_token(void *tiles, i64 pos, uint32_t v) {
    reinterpret_cast<T *>(tiles)[Tok<T>::index(pos)] = (T)v;
}

template <typename T>
__global__ void pack_bytes_kernel(const uint8_t *__restrict__ src, i64 n, void *tiles, i64 at) {
    const i64 g0 = at >> 5, g1 = (at + n + 31) >> 5;
    for (i64 g = g0 + (i64)blockIdx.x * blockDim.x + threadIdx.x; g < g1; g += (i64)gridDim.x * blockDim.x) {
        const i64 p = g * 32;
        const uint8_t *q = src + (p - at);
        if (p >= at && p + 32 <= at + n && ((uintptr_t)q & 15) == 0) {
            const uint4 x = __ldcs(reinterpret_cast<const uint4 *>(q)), y = __ldcs(reinterpret_cast<const uint4 *>(q) + 1);
            const uint32_t lo[4] = {x.x, x.y, x.z, x.w}, hi[4] = {y.x, y.y, y.z, y.w};
            uint4 *d = reinterpret_cast<uint4 *>(reinterpret_cast<T *>(tiles) + p);
            if (sizeof(T) == 2) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {  // word 4j + i = byte i of lo[j] | byte i of hi[j] << 16
                    const uint32_t a = __byte_perm(lo[j], 0, 0x4140), b = __byte_perm(lo[j], 0, 0x4342);
                    const uint32_t c = __byte_perm(hi[j], 0, 0x4140), e = __byte_perm(hi[j], 0, 0x4342);
                    d[j] = make_uint4(__byte_perm(a, c, 0x5410), __byte_perm(a, c, 0x7632), __byte_perm(b, e, 0x5410),
                                      __byte_perm(b, e, 0x7632));
                }
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const uint32_t w = j < 4 ? lo[j & 3] : hi[j & 3];
                    d[j] = make_uint4(w & 0xFFu, (w >> 8) & 0xFFu, (w >> 16) & 0xFFu, w >> 24);
                }
            }
        } else {
            for (int i = 0; i < 32; ++i)
                if (p + i >= at && p + i < at + n) put_token<T>(tiles, p + i, q[i]);
        }
    }
}

// ids must leave the top bit and the hole value free: out-of-range ids raise BAD_ID, ids that only a wider
// stream can hold NARROW (the host then widens the stream and packs again)
template <typename T>
struct PackedIds {
    unsigned int err = 0, largest = 0;
    __device__ __forceinline__ uint32_t operator()(int32_t v) {
        largest = max(largest, (unsigned int)v & STBPE_IDMASK);
        if (v < 0 || v == 0x7FFFFFFF)
            err |= STBPE_DERR_BAD_ID;
        else if ((uint32_t)v >= Tok<T>::IDMASK)
            err |= STBPE_DERR_NARROW;
        return (uint32_t)v & Tok<T>::IDMASK;
    }
};
// Bound by HBM (4 bytes read, 2 or 4 written per id).  Whole groups of the stream are written as 16-byte units, four per thread
// and turn with all loads in front, of 4 bytes each where the source is not 16-byte aligned; what lies before and behind them goes
// token by token.  (Append of 2^27 ids to 16- and 32-bit tokens: all token by token 379 and 454 us, now 176 and 219, from an unaligned
// source 187 and 231.)
template <typename T>
__global__ void __launch_bounds__(256) pack_ids_kernel(const int32_t *__restrict__ src, i64 n, void *tiles, i64 at, unsigned int *bad) {
    PackedIds<T> pack;
    const i64 head = min(n, (32 - (at & 31)) & 31), body = (n - head) & ~(i64)31;
    const i64 tid = (i64)blockIdx.x * blockDim.x + threadIdx.x, stride = (i64)gridDim.x * blockDim.x;
    auto units = [&](auto load) {  // load(i): the four ids from 4 i on
        constexpr int PER = 4, LOADS = sizeof(T) == 2 ? 2 : 1;  // units per turn; loads per unit
        uint4 *d = reinterpret_cast<uint4 *>(reinterpret_cast<T *>(tiles) + at + head);
        const i64 units = body / (4 * LOADS);
        for (i64 u0 = tid; u0 < units; u0 += PER * stride) {
            int4 x[PER][LOADS];
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                const i64 u = u0 + k * stride;
                if (u >= units) break;
                if (LOADS == 2) {  // unit j of a group: tokens 4j .. 4j + 3 and 16 + 4j .. 16 + 4j + 3
                    const i64 g = (u >> 2) * 8 + (u & 3);
                    x[k][0] = load(g), x[k][LOADS - 1] = load(g + 4);
                } else {
                    x[k][0] = load(u);
                }
            }
#pragma unroll
            for (int k = 0; k < PER; ++k) {
                const i64 u = u0 + k * stride;
                if (u >= units) break;
                const int4 lo = x[k][0];
                uint4 w = make_uint4(pack(lo.x), pack(lo.y), pack(lo.z), pack(lo.w));
                if (LOADS == 2) {
                    const int4 hi = x[k][LOADS - 1];
                    w.x |= pack(hi.x) << 16, w.y |= pack(hi.y) << 16, w.z |= pack(hi.z) << 16, w.w |= pack(hi.w) << 16;
                }
                d[u] = w;
            }
        }
    };
    const int32_t *q = src + head;
    if (((uintptr_t)q & 15) == 0)
        units([&](i64 i) { return __ldcs(reinterpret_cast<const int4 *>(q) + i); });
    else
        units([&](i64 i) { return make_int4(__ldcs(q + 4 * i), __ldcs(q + 4 * i + 1), __ldcs(q + 4 * i + 2), __ldcs(q + 4 * i + 3)); });
    for (i64 k = tid; k < n - body; k += stride) {
        const i64 i = k < head ? k : k + body;
        put_token<T>(tiles, at + i, pack(__ldcs(src + i)));
    }
    if (pack.err) atomicOr(bad, pack.err);
    __shared__ unsigned int s_largest[8];
    const unsigned int largest = __reduce_max_sync(0xFFFFFFFFu, pack.largest);
    if ((threadIdx.x & 31) == 0) s_largest[threadIdx.x >> 5] = largest;
    __syncthreads();
    if (threadIdx.x < 32) {
        const unsigned int all = __reduce_max_sync(0xFFFFFFFFu, threadIdx.x < 8 ? s_largest[threadIdx.x] : 0u);
        if (threadIdx.x == 0) atomicMax(bad + 1, all);  // DevState::max_id
    }
}

template <typename T>
__global__ void mark_row_starts_kernel(const i64 *__restrict__ off, i64 n_rows, void *tiles, i64 at) {
    const i64 r = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (r < n_rows && off[r] < off[r + 1]) {
        T *t = reinterpret_cast<T *>(tiles) + Tok<T>::index(at + off[r]);
        *t = (T)(*t | Tok<T>::FLAG);
    }
}

// records of a dense stream; the positions of the last tile past its end become holes
template <typename T>
__global__ void init_recs_kernel(EngineDev e, i64 n_tokens) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= e.n_tiles) return;
    T *tok = tile_ptr<T>(e, t);
    const i64 rem = n_tokens - (i64)t * STBPE_TILE;
    const int len = rem >= STBPE_TILE ? STBPE_TILE : (int)rem;
    for (int i = len; i < STBPE_TILE; ++i) tok[Tok<T>::index(i)] = (T)Tok<T>::HOLE;
    TileRec r;
    r.ver = 0;
    r.len = len;
    for (int i = 0; i < 3; ++i) r.head[i] = i < len ? Tok<T>::widen(tok[Tok<T>::index(i)]) : STBPE_NONE;
    r.tail = len > 0 ? Tok<T>::widen(tok[Tok<T>::index(len - 1)]) : STBPE_NONE;
    r.tail2 = len > 1 ? Tok<T>::widen(tok[Tok<T>::index(len - 2)]) : STBPE_NONE;
    r.pad = 0;
    e.recs[2 * t] = r;
    r.ver = -1;
    r.len = 0;
    e.recs[2 * t + 1] = r;
    e.tile_live[t] = (unsigned int)len;
}

__global__ void init_state_kernel(EngineDev e, int base_vocab, i64 n_tokens) {
    DevState h = {};
    h.base_vocab = base_vocab;
    h.n_live = n_tokens;
    *e.st = h;
}

__global__ void clear_table_kernel(EngineDev e) {
    u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x;
    u64 stride = (u64)gridDim.x * blockDim.x;
    for (; i <= e.mask; i += stride) {
        Slot s;
        s.key = STBPE_EMPTY;
        s.count = 0;
        e.table[i] = s;
    }
}

// ---------------------------------------------------------------------------------------
// K2  full adjacent-pair histogram of any stream (gpu_tokenizer/utils.py:558-635 without the sort): one warp
// per tile, one group of tokens per lane; every countable pair adds +1 into the CTA's shared-memory
// table, flushed at the end into the pair table (or, multi-GPU, into the rank-local delta table).
// ---------------------------------------------------------------------------------------
#define STBPE_COUNT_THREADS 512
#define STBPE_COUNT_SLOTS 8192
template <typename T, bool MG>
__global__ void __launch_bounds__(STBPE_COUNT_THREADS, 2) count_kernel(const __grid_constant__ EngineDev e) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    SmemTable tab;
    tab.keys = reinterpret_cast<u64 *>(smem_raw);
    tab.vals = reinterpret_cast<int *>(smem_raw + STBPE_COUNT_SLOTS * sizeof(u64));
    tab.mask = STBPE_COUNT_SLOTS - 1;
    smem_table_clear(tab);
    __syncthreads();
    const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    for (i64 t = (i64)blockIdx.x * warps + (threadIdx.x >> 5); t < e.n_tiles; t += (i64)gridDim.x * warps) {
        uint32_t w[Tok<T>::VEC * 4];
        load_group<T>(e, (int)t, lane, w);
        const uint32_t nxt = first_after(e, (int)t, 0x7FFFFFFF);
        for_each_pair<T>(w, live_mask<T>(w), lane, nxt, [&](uint32_t t0, uint32_t t1) {
            if (!(t1 & STBPE_FLAG)) smem_table_add<MG>(tab, e, ((u64)(t0 & STBPE_IDMASK) << 32) | (u64)t1, 1);
        });
    }
    __syncthreads();
    smem_table_flush<MG>(tab, e);
}

// ---------------------------------------------------------------------------------------
// K2, byte-level fast path.  Right after a load of bytes the stream is dense (every tile full)
// and every id is below 256, so a pair key fits 16 bits and the whole histogram fits a CTA's
// shared memory as 65 536 16-bit counters (two per 32-bit word, 128 KB).  Each token costs one
// shared-memory atomic on a direct index: no hashing, no key compare.
// A 16-bit counter is kept below 2^15: the thread whose add takes it to 0x8000 moves 0x8000 of it
// to the global 64-bit counter.  Should a counter ever be seen above 0xC000 (16 384 further
// adds would have to slip in before that subtraction lands) the kernel raises
// STBPE_DERR_DENSE_OVERFLOW and the host recounts with the general kernel, so the result is exact
// or the failure is reported, never silently wrong.
// ---------------------------------------------------------------------------------------
// Word of the shared-memory table that holds the counter of a 16-bit key (two counters per word).
// The bank would be bits 1-5 of the right byte alone, and text concentrates those on a dozen values
// (lower-case letters, the space), so the low five bits are XOR-ed with the low bits of the left
// byte: a bijection inside each left-byte row that spreads hot right bytes over the banks.
__device__ __forceinline__ unsigned int dense_word(unsigned int key) { return (key >> 1) ^ ((key >> 8) & 31u); }

// rare path of dense_add: the add took one of the two 16-bit halves of the word to 0x8000 or beyond
__device__ __noinline__ void dense_hand_over(unsigned int *s_tab, u64 *g_dense, unsigned int *derr,
                                             unsigned int key, unsigned int now) {
    const unsigned int sh = (key & 1u) * 16u;
    const unsigned int h = (now >> sh) & 0xFFFFu;  // this key's counter after the add
    if (h == 0x8000u) {
        atomicSub(&s_tab[dense_word(key)], 0x8000u << sh);
        atomicAdd(&g_dense[key], 0x8000ull);
    } else if (h > 0xC000u) {
        atomicOr(derr, STBPE_DERR_DENSE_OVERFLOW);
    }
    // 0x8000 < h <= 0xC000: another thread is handing this counter over; h < 0x8000: it was the other half
}

// t1 is below 256: a right-hand token that starts no row
__device__ __forceinline__ void dense_add(unsigned int *s_tab, u64 *g_dense, unsigned int *derr, uint32_t t0,
                                          uint32_t t1) {
    // key = (low byte of t0) << 8 | t1; bytes 1 and 2 of t1 are zero
    const unsigned int key = __byte_perm(t1, t0, 0x2140);
    const unsigned int inc = (key & 1u) ? 0x10000u : 1u;
    const unsigned int now = atomicAdd(&s_tab[dense_word(key)], inc) + inc;
    if (now & 0x80008000u) dense_hand_over(s_tab, g_dense, derr, key, now);
}

#define STBPE_DENSE_THREADS 1024
#define STBPE_DENSE_UNROLL 4
template <typename T>
__global__ void __launch_bounds__(STBPE_DENSE_THREADS, 1)
    count_dense_kernel(EngineDev e, u64 *g_dense) {
    extern __shared__ __align__(16) unsigned int s_tab[];  // 32 768 words
    for (int i = threadIdx.x; i < 32768; i += STBPE_DENSE_THREADS) s_tab[i] = 0u;
    __syncthreads();
    unsigned int *derr = &e.st->error;
    const uint4 *units = reinterpret_cast<const uint4 *>(e.tiles);
    const i64 n_units = (i64)e.n_tiles * (STBPE_TILE * sizeof(T) / 16);
    const i64 step = (i64)gridDim.x * STBPE_DENSE_THREADS * STBPE_DENSE_UNROLL;
    for (i64 base = (i64)blockIdx.x * STBPE_DENSE_THREADS * STBPE_DENSE_UNROLL; base < n_units; base += step) {
        uint4 v[STBPE_DENSE_UNROLL];
        uint32_t nx[STBPE_DENSE_UNROLL];
        load_unit_batch<T, STBPE_DENSE_UNROLL, STBPE_DENSE_THREADS>(units, base, n_units, v, nx);
#pragma unroll
        for (int u = 0; u < STBPE_DENSE_UNROLL; ++u)
            unit_pairs<T>(v[u], nx[u], [&](uint32_t t0, uint32_t t1) {
                if (!(t1 & Tok<T>::FLAG)) dense_add(s_tab, g_dense, derr, t0, t1);
            });
    }
    __syncthreads();
    for (int p = threadIdx.x; p < 32768; p += STBPE_DENSE_THREADS) {
        const unsigned int x = s_tab[p];
        const unsigned int w = (unsigned int)p ^ (((unsigned int)p >> 7) & 31u);  // inverse of dense_word
        if (x & 0xFFFFu) atomicAdd(&g_dense[2 * w], (u64)(x & 0xFFFFu));
        if (x >> 16) atomicAdd(&g_dense[2 * w + 1], (u64)(x >> 16));
    }
}

// Insert a key that is known to be absent (every directly indexed counter is its own key, and the
// table was cleared before the count): one compare-and-swap claims the slot, the count is a plain
// store, and nothing is marked dirty because a full refresh follows the initial count.
__device__ __forceinline__ bool table_insert_unique(const EngineDev &e, u64 key, i64 count) {
    u64 h = slot_of(e, key);
    for (unsigned int probe = 0; probe_on(e, probe); ++probe) {
        Slot *s = &e.table[h];
        if (atomicCAS(&s->key, STBPE_EMPTY, key) == STBPE_EMPTY) {
            s->count = count;
            return true;
        }
        h = (h + 1) & e.mask;
    }
    atomicOr(&e.st->error, STBPE_DERR_TABLE_FULL);
    return false;
}

// keys with a count from a smaller table into this one (grow_table)
__global__ void rehash_kernel(EngineDev e, const Slot *__restrict__ old, u64 n) {
    unsigned int moved = 0;
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (u64)gridDim.x * blockDim.x) {
        const Slot s = old[i];
        if (s.key != STBPE_EMPTY && s.count != 0 && table_insert_unique(e, s.key, s.count)) ++moved;
    }
    moved = __reduce_add_sync(0xFFFFFFFFu, moved);
    if ((threadIdx.x & 31) == 0 && moved) atomicAdd(&e.st->n_keys, (u64)moved);
}

#include "wide_count.cuh"

// dense 16-bit keys -> entries of the pair table (or of the rank-local delta table), and the largest id of a pair
template <bool MG>
__global__ void __launch_bounds__(256) dense_to_table_kernel(EngineDev e, const u64 *g_dense) {
    const int k = blockIdx.x * 256 + threadIdx.x;  // 256 CTAs: every counter has its thread
    const u64 c = g_dense[k];
    if (c) sink_add<MG>(e, ((u64)(k >> 8) << 32) | (u64)(k & 0xFF), (i64)c);
    const unsigned int largest = __reduce_max_sync(0xFFFFFFFFu, c ? (unsigned int)max(k >> 8, k & 0xFF) : 0u);
    if ((threadIdx.x & 31) == 0 && largest) atomicMax(&e.st->max_id, largest);
}

// ---------------------------------------------------------------------------------------
// K4  arg-max: block maxima refresh + reduction with the reference's tie-break
// ---------------------------------------------------------------------------------------
// maximum of one block, by one warp: its entry with the largest count, ties to the smaller key
__device__ __forceinline__ Slot block_max(const EngineDev &e, unsigned int blk, int lane) {
    const Slot *base = e.table + ((u64)blk << e.blk_shift);
    Slot best;
    best.key = STBPE_EMPTY;
    best.count = 0;
#pragma unroll 8
    for (int q = lane; q < (1 << e.blk_shift); q += 32) {
        const Slot x = ldcg_slot(base + q);
        if (x.key != STBPE_EMPTY && x.count > 0 && better(x.key, x.count, best.key, best.count)) best = x;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        Slot o;
        o.key = __shfl_down_sync(0xFFFFFFFFu, best.key, d);
        o.count = __shfl_down_sync(0xFFFFFFFFu, best.count, d);
        if (better(o.key, o.count, best.key, best.count)) best = o;
    }
    return best;
}

// recompute the maxima of the dirty blocks (or of all blocks), one warp per word of the bitmap / per block
__global__ void refresh_kernel(EngineDev e, int all) {
    const unsigned int lane = threadIdx.x & 31;
    const unsigned int w0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    if (all) {
        for (unsigned int blk = w0; blk < e.n_blocks; blk += nw) {
            const Slot s = block_max(e, blk, lane);
            if (lane == 0) e.blockmax[blk] = s;
        }
        for (unsigned int w = blockIdx.x * blockDim.x + threadIdx.x; w < (e.n_blocks + 31) / 32; w += gridDim.x * blockDim.x)
            e.dirty_bits[w] = 0u;
        return;
    }
    for (unsigned int w = w0; w < (e.n_blocks + 31) / 32; w += nw) {
        unsigned int bits = __ldcg(&e.dirty_bits[w]);
        if (!bits) continue;
        __syncwarp();
        if (lane == 0) e.dirty_bits[w] = 0u;
        for (; bits; bits &= bits - 1u) {
            const unsigned int blk = w * 32 + __ffs(bits) - 1;
            const Slot s = block_max(e, blk, lane);
            if (lane == 0) e.blockmax[blk] = s;
        }
    }
}

static __device__ __noinline__ i64 find_slot(const EngineDev &e, u64 key) {
    u64 h = slot_of(e, key);
    for (unsigned int probe = 0; probe < e.max_probe; ++probe) {
        const u64 k = *(volatile u64 *)&e.table[h].key;
        if (k == key) return (i64)h;
        if (k == STBPE_EMPTY) return -1;
        h = (h + 1) & e.mask;
    }
    return -1;
}

// Bookkeeping of one selected merge (gpu_tokenizer/bpe_trainer.py:4358-4373): log it, make it
// current, zero its table entry (no (a,b) pair survives its own merge).
__device__ __forceinline__ void begin_merge(const EngineDev &e, u64 key, i64 count, int new_id,
                                            bool may_be_absent) {
    DevState *st = e.st;
    const int mnum = st->merges_done;
    e.merges[2 * mnum] = (int32_t)(key >> 32);
    e.merges[2 * mnum + 1] = (int32_t)(key & 0xFFFFFFFFull);
    e.merge_counts[mnum] = count;
    e.live_before[mnum] = st->n_live;
    st->cur_a = (int)(key >> 32);
    st->cur_b = (int)(key & 0xFFFFFFFFull);
    st->cur_new = new_id;
    st->cur_count = count;
    st->merges_done = mnum + 1;
    st->n_work = 0;
    const i64 h = find_slot(e, key);
    if (h >= 0) {
        e.table[h].count = 0;
        if (e.world > 1) mark_dirty(e, (u64)h);
    } else if (!may_be_absent) {
        atomicOr(&st->error, STBPE_DERR_KEY_MISSING);
    }
}

// ---------------------------------------------------------------------------------------
// Candidate list (one rank).  A new threshold is found by a histogram of the table over 2048 buckets in
// selection order: first logarithmic in the count (5 bits below the leading one), then, should one bucket
// hold too many pairs (ties late in a run, very flat histograms), linear inside that bucket, first over its
// counts and, when a single count is left, over the keys.
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ int log_bucket(i64 c) {  // monotone in c >= 1
    if (c < 64) return (int)c;
    const int lg = 63 - __clzll(c);
    return 64 + (lg - 6) * 32 + (int)((c >> (lg - 5)) & 31);
}
__device__ __forceinline__ i64 log_bucket_low(int b) {
    if (b < 64) return b;
    const int lg = (b - 64) / 32 + 6;
    return ((i64)(32 + ((b - 64) & 31))) << (lg - 5);
}
// width of a linear bucket over [lo, hi]: a power of two that needs at most STBPE_CAND_BUCKETS of them
__device__ __forceinline__ int linear_shift(u64 lo, u64 hi) {
    int sh = 0;
    while (((hi - lo) >> sh) >= STBPE_CAND_BUCKETS) ++sh;
    return sh;
}

// a fresh count: no list, and no add is admitted to one
__global__ void cand_none_kernel(EngineDev e) {
    e.st->cand_state = STBPE_CAND_NONE;
    e.st->n_cand = 0;
    e.st->theta_count = 0x7FFFFFFFFFFFFFFFll;
    e.st->theta_key = 0;
    e.st->peek_valid = 0;
}

// pass over the table; larger bucket = earlier in selection order
__global__ void __launch_bounds__(512) cand_hist_kernel(EngineDev e) {
    __shared__ unsigned int s_h[STBPE_CAND_BUCKETS];
    const DevState *st = e.st;
    const bool refine = st->cand_state == STBPE_CAND_REFINE;
    const i64 lo = st->refine_lo, hi = st->refine_hi;
    const u64 klo = st->refine_klo, khi = st->refine_khi;
    const bool by_key = refine && lo == hi;
    const int sh = !refine ? 0 : (by_key ? linear_shift(klo, khi) : linear_shift((u64)lo, (u64)hi));
    for (int i = threadIdx.x; i < STBPE_CAND_BUCKETS; i += blockDim.x) s_h[i] = 0u;
    __syncthreads();
#pragma unroll 4
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i <= e.mask; i += (u64)gridDim.x * blockDim.x) {
        const Slot s = ldcg_slot(e.table + i);
        if (s.key == STBPE_EMPTY || s.count <= 0) continue;
        int b;
        if (!refine) {
            b = log_bucket(s.count);
        } else if (by_key) {
            if (s.count != lo || s.key < klo || s.key > khi) continue;
            b = (int)((khi - s.key) >> sh);
        } else {
            if (s.count < lo || s.count > hi) continue;
            b = (int)((u64)(s.count - lo) >> sh);
        }
        atomicAdd(&s_h[b], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < STBPE_CAND_BUCKETS; i += blockDim.x)
        if (s_h[i]) atomicAdd(&e.cand_hist[i], s_h[i]);
}

// The threshold out of the histogram (which is left zeroed for the next search): buckets are taken from the top
// while the list stays within STBPE_CAND_MOST; with too few taken and the next one too large, that bucket
// is searched again (STBPE_CAND_REFINE).
// (One thread walking down the 2048 buckets took up to 30 us; the running sums of a block scan take 2.)
__global__ void __launch_bounds__(1024) cand_decide_kernel(EngineDev e, u64 key_hi) {
    static_assert(STBPE_CAND_BUCKETS == 2 * 1024, "two buckets per thread");
    __shared__ i64 s_sum[32];
    __shared__ int s_first;   // place from the top of the first bucket that does not fit
    __shared__ i64 s_taken;   // pairs in the buckets above it
    DevState *st = e.st;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, hi_b = STBPE_CAND_BUCKETS - 1 - 2 * (int)threadIdx.x;
    const i64 n0 = e.cand_hist[hi_b], n1 = e.cand_hist[hi_b - 1], base = st->cand_state == STBPE_CAND_REFINE ? st->refine_above : 0;
    e.cand_hist[hi_b] = e.cand_hist[hi_b - 1] = 0u;
    if (threadIdx.x == 0) s_first = STBPE_CAND_BUCKETS;
    i64 incl = n0 + n1;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const i64 o = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= d) incl += o;
    }
    if (lane == 31) s_sum[warp] = incl;
    __syncthreads();
    i64 before = base + incl - n0 - n1;
    for (int w = 0; w < warp; ++w) before += s_sum[w];
    const bool out0 = before + n0 > STBPE_CAND_MOST, out1 = before + n0 + n1 > STBPE_CAND_MOST;
    if (out0 || out1) atomicMin(&s_first, 2 * (int)threadIdx.x + (out0 ? 0 : 1));
    __syncthreads();
    if (s_first == 2 * (int)threadIdx.x) s_taken = before;
    if (s_first == 2 * (int)threadIdx.x + 1) s_taken = before + n0;
    if (s_first == STBPE_CAND_BUCKETS && threadIdx.x == 1023) s_taken = before + n0 + n1;
    __syncthreads();
    if (threadIdx.x != 0) return;
    st->n_cand = 0;
    const bool refine = st->cand_state == STBPE_CAND_REFINE;
    const i64 lo = st->refine_lo, hi = st->refine_hi;
    const u64 klo = st->refine_klo, khi = st->refine_khi;
    const bool by_key = refine && lo == hi;
    const int sh = !refine ? 0 : (by_key ? linear_shift(klo, khi) : linear_shift((u64)lo, (u64)hi));
    const i64 taken = s_taken;
    const int b = STBPE_CAND_BUCKETS - 1 - s_first;
    // bucket b does not fit (or b < 0: everything does); the list takes the buckets above it
    if (b >= 0 && taken < STBPE_CAND_LEAST) {
        st->cand_state = STBPE_CAND_REFINE;
        st->refine_above = taken;
        if (by_key) {
            st->refine_khi = khi - ((u64)b << sh);
            const u64 w = (1ull << sh) - 1;
            st->refine_klo = st->refine_khi - klo < w ? klo : st->refine_khi - w;
        } else if (refine) {
            st->refine_lo = lo + (i64)((u64)b << sh);
            const i64 top = st->refine_lo + (i64)(1ull << sh) - 1;
            st->refine_hi = top < hi ? top : hi;
            st->refine_klo = 0;
            st->refine_khi = key_hi;
        } else {
            st->refine_lo = log_bucket_low(b);
            st->refine_hi = log_bucket_low(b + 1) - 1;
            st->refine_klo = 0;
            st->refine_khi = key_hi;
        }
        return;
    }
    if (by_key) {  // the taken buckets hold the keys up to khi - ((b + 1) << sh)
        st->theta_count = lo;
        st->theta_key = khi - ((u64)(b + 1) << sh) + 1;
    } else {
        const i64 from = b < 0 && !refine ? 1 : (refine ? lo + (i64)((u64)(b + 1) << sh) : log_bucket_low(b + 1));
        st->theta_count = from - 1;  // the smallest count taken is `from`
        st->theta_key = 0;
    }
    st->cand_state = STBPE_CAND_READY;
}

__global__ void __launch_bounds__(512) cand_collect_kernel(EngineDev e) {
    if (e.st->cand_state != STBPE_CAND_READY) return;
    Theta t;
    t.count = e.st->theta_count, t.key = e.st->theta_key;
#pragma unroll 4
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i <= e.mask; i += (u64)gridDim.x * blockDim.x) {
        const Slot s = ldcg_slot(e.table + i);
        if (s.key != STBPE_EMPTY && s.count > 0 && t.admits(s.count, s.key)) {
            const unsigned int j = atomicAdd(&e.st->n_cand, 1u);
            if (j < STBPE_CAND_CAP) e.cand[j] = (unsigned int)i;
        }
    }
}

// stop rules of the loop: bpe_trainer.py:4304-4308 (no pairs), :2491-2494 / :4361-4364 (count < 2)
__device__ __forceinline__ void advance_or_stop(const EngineDev &e, u64 key, i64 count) {
    DevState *st = e.st;
    if (st->error) {
        st->stopped = 1;
        st->stop_reason = 4;
    } else if (st->merges_done >= st->target) {
        st->stopped = 1;
        st->stop_reason = 1;
    } else if (count <= 0) {
        st->stopped = 1;
        st->stop_reason = 2;
    } else if (count < 2) {
        st->stopped = 1;
        st->stop_reason = 3;
    } else {
        begin_merge(e, key, count, st->base_vocab + st->merges_done, e.world > 1);
    }
}

// best pair of the candidate list, by one CTA of 1024 threads (all threads get it); false when the list has run
// dry or over: the host then searches a new threshold and asks again
__device__ __forceinline__ bool best_candidate(const EngineDev &e, unsigned int n, Slot &best) {
    __shared__ u64 s_k[32];
    __shared__ i64 s_c[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    u64 bk = STBPE_EMPTY;
    i64 bc = 0;
    for (unsigned int i = threadIdx.x; i < min(n, STBPE_CAND_CAP); i += blockDim.x) {
        const Slot x = ldcg_slot(e.table + e.cand[i]);
        if (x.count > 0 && better(x.key, x.count, bk, bc)) bk = x.key, bc = x.count;
    }
#pragma unroll 1
    for (int level = 0; level < 2; ++level) {
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            const u64 ok = __shfl_xor_sync(0xFFFFFFFFu, bk, d);
            const i64 oc = __shfl_xor_sync(0xFFFFFFFFu, bc, d);
            if (better(ok, oc, bk, bc)) bk = ok, bc = oc;
        }
        if (level == 0) {
            if (lane == 0) s_k[warp] = bk, s_c[warp] = bc;
            __syncthreads();
            bk = s_k[lane], bc = s_c[lane];
        }
    }
    best.key = bk;
    best.count = bc;
    Theta t;
    t.count = e.st->theta_count, t.key = e.st->theta_key;
    return e.st->cand_state == STBPE_CAND_READY && n <= STBPE_CAND_CAP && (t.admits(bc, bk) || (bc <= 0 && t.count == 0));
}

// best pair as a peek into the state, or as the loop's next step
__global__ void __launch_bounds__(1024) choose_kernel(EngineDev e, int advance) {
    DevState *st = e.st;
    if (advance && st->stopped) return;
    Slot best;
    const bool valid = best_candidate(e, st->n_cand, best);
    if (threadIdx.x != 0) return;
    st->peek_valid = valid;
    st->peek_key = best.key;
    st->peek_count = best.count;
    if (advance && valid) advance_or_stop(e, best.key, best.count);
}

// Best count and the keys that hold it, behind the state (a key may appear twice: the list may name it twice).
// peek_ties = 0 when the list need not hold all of them (the threshold lies inside that count).
__global__ void __launch_bounds__(1024) ties_kernel(EngineDev e) {
    __shared__ int s_n;
    DevState *st = e.st;
    u64 *out = reinterpret_cast<u64 *>(reinterpret_cast<unsigned char *>(st) + STBPE_TIES_OFFSET);
    const unsigned int n = st->n_cand;
    if (threadIdx.x == 0) s_n = 0;
    Slot best;
    const bool valid = best_candidate(e, n, best);
    if (valid && best.count > st->theta_count) {
        for (unsigned int i = threadIdx.x; i < n; i += blockDim.x) {
            const Slot x = ldcg_slot(e.table + e.cand[i]);
            if (x.count == best.count && x.count > 0) {
                const int j = atomicAdd(&s_n, 1);
                if (j < STBPE_TIES_CAP) out[j] = x.key;
            }
        }
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    st->peek_valid = valid;
    st->peek_key = best.key;
    st->peek_count = best.count;
    st->peek_ties = s_n;
}

#define STBPE_SELECT_THREADS 256
__device__ __forceinline__ void block_best(u64 &bk, i64 &bc, u64 *s_k, i64 *s_c) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        const u64 ok = __shfl_down_sync(0xFFFFFFFFu, bk, d);
        const i64 oc = __shfl_down_sync(0xFFFFFFFFu, bc, d);
        if (better(ok, oc, bk, bc)) {
            bk = ok;
            bc = oc;
        }
    }
    if (lane == 0) {
        s_k[warp] = bk;
        s_c[warp] = bc;
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < STBPE_SELECT_THREADS / 32; ++w)
            if (better(s_k[w], s_c[w], bk, bc)) {
                bk = s_k[w];
                bc = s_c[w];
            }
    __syncthreads();
}

#include "peer_kernels.cuh"

// Best pair over all block maxima: every CTA reduces its share, the last one to finish reduces theirs.
// mode 0: peek (result into the state); 2: candidate of this rank into cand; 3: candidate of this rank into every
// peer mailbox, then wait for the peers' candidates and commit (target = the merge target of the engine)
__global__ void __launch_bounds__(STBPE_SELECT_THREADS)
    select_kernel(EngineDev e, int mode, Slot *partial, i64 *cand, int target = 0) {
    DevState *st = e.st;
    __shared__ u64 s_k[STBPE_SELECT_THREADS / 32];
    __shared__ i64 s_c[STBPE_SELECT_THREADS / 32];
    __shared__ int s_last;
    u64 bk = STBPE_EMPTY;
    i64 bc = 0;
#pragma unroll 4
    for (unsigned int i = blockIdx.x * STBPE_SELECT_THREADS + threadIdx.x; i < e.n_blocks; i += gridDim.x * STBPE_SELECT_THREADS) {
        const Slot x = ldcg_slot(e.blockmax + i);
        if (x.count > 0 && better(x.key, x.count, bk, bc)) bk = x.key, bc = x.count;
    }
    block_best(bk, bc, s_k, s_c);
    if (threadIdx.x == 0) {
        Slot x;
        x.key = bk;
        x.count = bc;
        partial[blockIdx.x] = x;
        __threadfence();
        s_last = (atomicAdd(&st->ticket, 1u) == gridDim.x - 1);
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    bk = STBPE_EMPTY;
    bc = 0;
    for (unsigned int i = threadIdx.x; i < gridDim.x; i += STBPE_SELECT_THREADS) {
        const Slot x = ldcg_slot(partial + i);
        if (x.count > 0 && better(x.key, x.count, bk, bc)) bk = x.key, bc = x.count;
    }
    block_best(bk, bc, s_k, s_c);
    if (threadIdx.x != 0) return;
    st->ticket = 0;
    if (mode == 0) {
        st->peek_key = bk;
        st->peek_count = bc;
    } else if (mode == 2) {
        cand[0] = (i64)bk;
        cand[1] = bc;
        cand[2] = st->round_incomplete;
        cand[3] = 0;
    } else {
        publish_candidate(e, bk, bc, st->round_incomplete);
        commit_from_mailbox(e, target);
    }
}

// ---------------------------------------------------------------------------------------
// Tile skipping.  A merge (a,b) changes a tile only if one of its tokens is half of a pair (a,b).  The pair
// filter records, per tile, the pairs that have a token in it (the pair across a seam is entered for
// both tiles), so
//     visit tile t  iff  all three filter rows of (a,b) have bit t set, or t is a wildcard tile.
// (Re)build from the stream: one CTA handles 32 consecutive tiles, i.e. one word of every row: it
// collects the bits in shared memory and then writes the group's words with plain stores.
// ---------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(1024) presence_rebuild_kernel(EngineDev e) {
    extern __shared__ unsigned int s_rows[];  // STBPE_PROWS words
    const int n_groups = (e.n_tiles + 31) / 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int grp = blockIdx.x; grp < n_groups; grp += gridDim.x) {
        for (int i = threadIdx.x; i < STBPE_PROWS; i += blockDim.x) s_rows[i] = 0u;
        __syncthreads();
        const int tile = grp * 32 + warp;  // blockDim.x == 1024: one warp per tile of the group
        if (tile < e.n_tiles) {
            auto enter = [&](uint32_t t0, uint32_t t1) {
                if (t1 & STBPE_FLAG) return;  // not a countable pair
                unsigned int r1, r2, r3;
                filter_rows(((u64)(t0 & STBPE_IDMASK) << 32) | (u64)t1, r1, r2, r3);
                atomicOr(&s_rows[r1], 1u << warp);
                atomicOr(&s_rows[r2], 1u << warp);
                atomicOr(&s_rows[r3], 1u << warp);
            };
            uint32_t w[Tok<T>::VEC * 4];
            load_group<T>(e, tile, lane, w);
            const uint32_t L = live_mask<T>(w);
            const uint32_t ne = __ballot_sync(0xFFFFFFFFu, L != 0u);
            if (ne) {
                for_each_pair<T>(w, L, lane, first_after(e, tile, 0x7FFFFFFF), enter);
                if (lane == __ffs(ne) - 1) {  // the pair that ends at this tile's first token
                    uint32_t first = STBPE_NONE;
#pragma unroll
                    for (int i = 31; i >= 0; --i)
                        if ((L >> i) & 1u) first = Tok<T>::get(w, i);
                    const uint32_t prev = last_before(e, tile, 0x7FFFFFFF);
                    if (prev != STBPE_NONE) enter(prev, first);
                }
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < STBPE_PROWS; i += blockDim.x)
            e.presence[(size_t)grp * STBPE_PPITCH + i] = s_rows[i];
        if (threadIdx.x == 0) e.presence[(size_t)grp * STBPE_PPITCH + STBPE_PROWS] = 0u;  // no wildcards
        __syncthreads();
    }
}

// number of keys that hold exactly `count` (tie statistics; full table scan, on demand only)
__global__ void count_ties_kernel(EngineDev e) {
    const i64 target = e.st->peek_count;
    i64 n = 0;
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i <= e.mask; i += (u64)gridDim.x * blockDim.x) {
        const Slot s = e.table[i];
        if (s.key != STBPE_EMPTY && s.count == target) ++n;
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) n += __shfl_down_sync(0xFFFFFFFFu, n, d);
    if ((threadIdx.x & 31) == 0 && n) atomicAdd((u64 *)&e.st->peek_ties, (u64)n);
}

// ---------------------------------------------------------------------------------------
// exports
// ---------------------------------------------------------------------------------------
// Entries with a count, unordered.  K = uint32_t: (a << 16) | b and a 32-bit count (ids and counts that fit).  A
// CTA reserves the places of its entries of a step at once.
template <typename K>
__global__ void __launch_bounds__(512) export_table_kernel(EngineDev e, K *keys, K *counts, i64 cap) {
    __shared__ int s_sum[16];
    __shared__ i64 s_base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int PER = 8;
    for (u64 i0 = (u64)blockIdx.x * 512 * PER; i0 <= e.mask; i0 += (u64)gridDim.x * 512 * PER) {
        Slot s[PER];
        int own = 0;
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const u64 i = i0 + (u64)k * 512 + threadIdx.x;
            s[k].key = STBPE_EMPTY, s[k].count = 0;
            if (i <= e.mask) s[k] = ldcg_slot(e.table + i);
            if (s[k].key == STBPE_EMPTY) s[k].count = 0;
            own += s[k].count != 0;
        }
        int incl = own;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int o = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (lane >= d) incl += o;
        }
        if (lane == 31) s_sum[warp] = incl;
        __syncthreads();
        if (threadIdx.x == 0) {
            int total = 0;
            for (int w = 0; w < 16; ++w) {
                const int x = s_sum[w];
                s_sum[w] = total;
                total += x;
            }
            s_base = total ? (i64)atomicAdd((u64 *)&e.st->export_n, (u64)total) : 0;
        }
        __syncthreads();
        i64 at = s_base + s_sum[warp] + incl - own;
#pragma unroll
        for (int k = 0; k < PER; ++k)
            if (s[k].count != 0) {
                if (at < cap) {
                    keys[at] = sizeof(K) == 4 ? (K)(((s[k].key >> 32) << 16) | (s[k].key & 0xFFFFull)) : (K)s[k].key;
                    counts[at] = (K)s[k].count;
                }
                ++at;
            }
        __syncthreads();
    }
}

__global__ void widen_entries_kernel(const uint32_t *__restrict__ k, const uint32_t *__restrict__ c, i64 n, u64 *__restrict__ keys, i64 *__restrict__ counts) {
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
        const uint32_t x = k[i];
        keys[i] = ((u64)(x >> 16) << 32) | (u64)(x & 0xFFFFu);
        counts[i] = (i64)c[i];
    }
}

// keys whose count equals `count` (unordered; the host sorts the few there are)
__global__ void export_ties_kernel(EngineDev e, i64 count, u64 *keys, i64 cap) {
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i <= e.mask; i += (u64)gridDim.x * blockDim.x) {
        const Slot s = e.table[i];
        if (s.key != STBPE_EMPTY && s.count == count) {
            const i64 j = (i64)atomicAdd((u64 *)&e.st->export_n, 1ull);
            if (j < cap) keys[j] = s.key;
        }
    }
}

// Live tokens of all tiles, in order, into a dense stream (tile_off = exclusive prefix of the live counts):
//   re-pack : after many merges a stream is full of holes, and every pass over it pays for them; also the step
//             from a 16-bit to a 32-bit stream (TD wider than TS)
//   export  : as int32 ids with bit 31 = row start, in stream order
// One warp per tile: the tile's live tokens are squeezed together in shared memory (rank = live tokens before
// it, from the lanes' masks), then stored 32 consecutive positions at a time.
#define STBPE_REPACK_THREADS 256
template <typename TS, typename TD, bool EXPORT>
__global__ void __launch_bounds__(STBPE_REPACK_THREADS) repack_copy_kernel(EngineDev e, const i64 *__restrict__ tile_off, TD *__restrict__ dst) {
    __shared__ TS s_tok[STBPE_REPACK_THREADS / 32][STBPE_TILE];
    const int warps = blockDim.x >> 5, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (i64 tile = (i64)blockIdx.x * warps + warp; tile < e.n_tiles; tile += (i64)gridDim.x * warps) {
        uint32_t w[Tok<TS>::VEC * 4];
        load_group<TS>(e, (int)tile, lane, w);
        const uint32_t L = live_mask<TS>(w);
        int incl = __popc(L);
        const int mine = incl;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int n = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (lane >= d) incl += n;
        }
        const int len = __shfl_sync(0xFFFFFFFFu, incl, 31);
        int r = incl - mine;
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 32; ++i)
            if ((L >> i) & 1u) s_tok[warp][r++] = (TS)(sizeof(TS) == 2 ? (i < 16 ? w[i] & 0xFFFFu : w[i & 15] >> 16) : w[i % (Tok<TS>::VEC * 4)]);
        __syncwarp();
        const i64 o = tile_off[tile];
        for (int i = lane; i < len; i += 32) {
            const uint32_t c = Tok<TS>::widen(s_tok[warp][i]);
            if (EXPORT)
                dst[o + i] = (TD)c;
            else
                dst[Tok<TD>::index(o + i)] = (TD)Tok<TD>::narrow(c);
        }
    }
}

// a stream that is still being loaded, token by token into the wider format
__global__ void widen_copy_kernel(const uint16_t *__restrict__ src, uint32_t *__restrict__ dst, i64 n) {
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x)
        dst[i] = Tok<uint16_t>::widen(src[Tok<uint16_t>::index(i)]);
}

__global__ void tile_lens_kernel(EngineDev e, i64 *lens) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < e.n_tiles) lens[t] = (i64)e.tile_live[t];
}

// ---------------------------------------------------------------------------------------
// multi-GPU: drain the rank-local delta table into per-owner outbox chunks; apply an inbox
// ---------------------------------------------------------------------------------------
// chunk headers start a round at zero: done once when the buffers are set and after every exchange
// (apply_inbox_kernel), so a round needs no separate reset launch
__global__ void outbox_reset_kernel(EngineDev e) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < e.world) {
        Slot h;
        h.key = 0;
        h.count = 0;
        e.outbox[(i64)p * (e.cap_per_peer + 1)] = h;
    }
    if (p == 0) {
        e.st->n_lkept = 0;
        e.st->round_incomplete = 0;
    }
}

// Move the rank-local deltas into the per-owner outbox chunks.  A chunk holds cap_per_peer
// entries; what does not fit stays in the local table and is listed again for the next round
// (the header count of a chunk keeps counting past the capacity, which tells the receiver that
// more is to come).
__global__ void drain_ltable_kernel(EngineDev e) {
    __shared__ int s_last;
    const unsigned int n = e.st->n_ltouched;
    unsigned int *kept = e.ltouched + (e.lmask + 1);
    for (unsigned int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned int idx = e.ltouched[i];
        Slot *s = &e.ltable[idx];
        const Slot v = *s;
        if (v.count != 0) {
            const int owner = owner_of(v.key, e.world);
            Slot *chunk = e.outbox + (i64)owner * (e.cap_per_peer + 1);
            const i64 j = (i64)atomicAdd(&chunk[0].key, 1ull);
            if (j >= e.cap_per_peer) {
                kept[atomicAdd(&e.st->n_lkept, 1u)] = idx;
                e.st->round_incomplete = 1;
                continue;
            }
            chunk[1 + j] = v;
        }
        s->key = STBPE_EMPTY;
        s->count = 0;
    }
    // the last CTA to finish turns the kept entries into the list the next inserts append to
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = (atomicAdd(&e.st->ticket, 1u) == gridDim.x - 1);
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const unsigned int nk = *(volatile unsigned int *)&e.st->n_lkept;
    for (unsigned int i = threadIdx.x; i < nk; i += blockDim.x) e.ltouched[i] = ((volatile unsigned int *)kept)[i];
    __syncthreads();
    if (threadIdx.x == 0) {
        e.st->n_ltouched = nk;
        e.st->n_lkept = 0;
        e.st->ticket = 0;
    }
}

__global__ void apply_inbox_kernel(EngineDev e) {
    if (blockIdx.x == 0 && threadIdx.x < e.world) {  // the exchange is over: headers for the next round
        Slot h;
        h.key = 0;
        h.count = 0;
        e.outbox[(i64)threadIdx.x * (e.cap_per_peer + 1)] = h;
    }
    unsigned int fresh = 0;
    for (int p = 0; p < e.world; ++p) {
        const Slot *chunk = e.inbox + (i64)p * (e.cap_per_peer + 1);
        i64 n = (i64)chunk[0].key;
        if (n > e.cap_per_peer) {
            n = e.cap_per_peer;
            if (blockIdx.x == 0 && threadIdx.x == 0) e.st->round_incomplete = 1;
        }
        for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
            const Slot v = chunk[1 + i];
            table_add<NOTE_DIRTY>(e, v.key, v.count, false, fresh);
        }
    }
    if (fresh) atomicAdd(&e.st->n_keys, (u64)fresh);
}

// Every rank evaluates the same gathered candidates {key, count, incomplete, -} and reaches the
// same decision: if any rank still has deltas in flight the next round only exchanges, otherwise
// the best candidate (highest count, smallest key) is committed or a stop rule fires.
__global__ void commit_kernel(EngineDev e, const i64 *all_cands, int target) {
    DevState *st = e.st;
    st->target = target;
    st->round_incomplete = 0;  // the candidates carried this round's flag; the next round starts clean
    if (st->stopped) return;
    u64 bk = STBPE_EMPTY;
    i64 bc = 0;
    bool incomplete = false;
    for (int r = 0; r < e.world; ++r) {
        const u64 k = (u64)all_cands[4 * r];
        const i64 c = all_cands[4 * r + 1];
        incomplete |= all_cands[4 * r + 2] != 0;
        if (c > 0 && better(k, c, bk, bc)) {
            bk = k;
            bc = c;
        }
    }
    if (incomplete) {
        st->exchange_only = 1;
        return;
    }
    st->exchange_only = 0;
    advance_or_stop(e, bk, bc);
}
