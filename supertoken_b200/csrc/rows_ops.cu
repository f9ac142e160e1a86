// Stateless operators on padded [B, L] batches, with the reference's operator signatures
// (gpu_tokenizer/utils.py:691-706 count_pairs, :413-555 apply_merge_once).
#include <cub/device/device_radix_sort.cuh>
#include <cuda_runtime.h>

#include <cstdio>
#include <mutex>
#include <string>

#include "../../include/stbpe.h"
#include "block_cache.h"
#include "common.cuh"

#define STBPE_VISIBLE __attribute__((visibility("default")))
#define ROWS_NT 256
#define ROWS_IPT 8
#define ROWS_CHUNK (ROWS_NT * ROWS_IPT)
#define ROWS_BYTE_PAIRS 65536

namespace {

struct RowsTable {
    Slot *table;
    u64 mask;
    unsigned int *error;
    u64 *n_keys;
    u64 *bytes;  // large batches: counters of the pairs of two ids below 256, which are not in the table; else null
};

__device__ __forceinline__ void rows_table_add(const RowsTable &t, u64 key) {
    u64 h = mix64(key) & t.mask;
    for (u64 probe = 0; probe <= t.mask; ++probe) {
        Slot *s = &t.table[h];
        u64 k = *(volatile u64 *)&s->key;
        if (k == STBPE_EMPTY) {
            u64 old = atomicCAS(&s->key, STBPE_EMPTY, key);
            if (old == STBPE_EMPTY) {
                atomicAdd(t.n_keys, 1ull);
                k = key;
            } else {
                k = old;
            }
        }
        if (k == key) {
            atomicAdd((u64 *)&s->count, 1ull);
            return;
        }
        h = (h + 1) & t.mask;
    }
    atomicOr(t.error, 1u);
}

__global__ void rows_clear_kernel(RowsTable t) {
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i <= t.mask; i += (u64)gridDim.x * blockDim.x) {
        Slot s;
        s.key = STBPE_EMPTY;
        s.count = 0;
        t.table[i] = s;
    }
}

// a pair (i, i+1) counts when both positions are valid (gpu_tokenizer/utils.py:586)
__global__ void rows_count_kernel(const int32_t *__restrict__ tokens, const uint8_t *__restrict__ valid,
                                  i64 B, i64 L, RowsTable t) {
    const i64 width = L - 1, total = B * width;
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (i64)gridDim.x * blockDim.x) {
        const i64 r = i / width, c = i - r * width;
        const i64 p = r * L + c;
        if (valid[p] && valid[p + 1])
            rows_table_add(t, ((u64)(uint32_t)tokens[p] << 32) | (u64)(uint32_t)tokens[p + 1]);
    }
}

// (also the byte pairs, which then count among the keys)
__global__ void rows_export_kernel(RowsTable t, u64 *keys, i64 *counts, u64 *n_out, i64 cap) {
    const u64 slots = (t.mask | 31u) + 1, all = slots + (t.bytes ? ROWS_BYTE_PAIRS : 0);  // whole warps
    const int lane = threadIdx.x & 31;
    for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < all; i += (u64)gridDim.x * blockDim.x) {
        Slot s;
        s.key = STBPE_EMPTY, s.count = 0;
        if (i <= t.mask) {
            s = t.table[i];
        } else if (i >= slots) {
            const u64 k = i - slots;
            s.count = (i64)t.bytes[k];
            if (s.count) s.key = ((k >> 8) << 32) | (k & 0xFFull);
        }
        const bool have = s.key != STBPE_EMPTY;
        const unsigned int who = __ballot_sync(0xFFFFFFFFu, have);
        if (!who) continue;
        u64 at = 0;
        if (lane == 0) {
            at = atomicAdd(n_out, (u64)__popc(who));
            if (i >= slots) atomicAdd(t.n_keys, (u64)__popc(who));
        }
        at = __shfl_sync(0xFFFFFFFFu, at, 0) + __popc(who & ((1u << lane) - 1u));
        if (have && (i64)at < cap) {
            keys[at] = s.key;
            counts[at] = s.count;
        }
    }
}

// unique (a, b) rows ascending, unused rows -1 / 0, length (gpu_tokenizer/utils.py:622-635)
__global__ void rows_write_kernel(const u64 *__restrict__ keys, const i64 *__restrict__ counts, i64 n,
                                  int32_t *pair_keys, i64 *pair_counts, i64 cap, i64 *length) {
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < cap; i += (i64)gridDim.x * blockDim.x) {
        if (i < n) {
            pair_keys[2 * i] = (int32_t)(keys[i] >> 32);
            pair_keys[2 * i + 1] = (int32_t)(keys[i] & 0xFFFFFFFFull);
            pair_counts[i] = counts[i];
        } else {
            pair_keys[2 * i] = -1;
            pair_keys[2 * i + 1] = -1;
            pair_counts[i] = 0;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0 && length) *length = n;
}

// ---- stbpe_rows_count_pairs
// Threads and shared-memory slots of a counting CTA.  Small batches: short to clear, and several CTAs per SM.  From 2^18
// cells on a kernel with one CTA per SM (a pair that finds no slot is added in L2 by
// itself: with 2048 slots 2048 x 4096 cells of mixed text, 6 900 pairs, took 181 us).
#define ROWS_SMALL_NT 256
#define ROWS_SMALL_SLOTS 2048
#define ROWS_LARGE_NT 1024
#define ROWS_LARGE_SLOTS 16384  // of a CTA whose pairs are mostly not of bytes ...
#define ROWS_MIXED_SLOTS 8192   // ... and beside the byte pairs' counters
#define ROWS_LARGE_SMEM (ROWS_BYTE_PAIRS * 2 + ROWS_MIXED_SLOTS * 12)
static_assert(ROWS_LARGE_SLOTS * 12 <= ROWS_LARGE_SMEM, "either layout fits");
#define ROWS_LARGE_CELLS (1 << 18)
#define ROWS_DIRECT_CELLS (1 << 16)
#define ROWS_RANK_MAX 16384   // up to this many pairs are sorted by counting smaller keys, two launches instead of a radix sort's nine
#define ROWS_RANK_TILE 512

__global__ void rows_init_kernel(RowsTable t, unsigned int *rank, unsigned int n_rank) {
    const u64 first = (u64)blockIdx.x * blockDim.x + threadIdx.x, step = (u64)gridDim.x * blockDim.x;
    Slot s;
    s.key = STBPE_EMPTY;
    s.count = 0;
    for (u64 i = first; i <= t.mask; i += step) t.table[i] = s;
    for (u64 i = first; i < n_rank; i += step) rank[i] = 0u;
    if (t.bytes)
        for (u64 i = first; i < ROWS_BYTE_PAIRS; i += step) t.bytes[i] = 0;
    if (first < 3) t.n_keys[first] = 0;  // number of keys, error, export cursor
}

// key + n into the table; a table that fills up ends the count (the host repeats it with a larger one).  Only the number of
// keys says that it is full: a table of twice as many slots as the batch has pairs may well hold 64 keys side by side.
__device__ __forceinline__ void rows_add(const RowsTable &t, u64 key, u64 n) {
    u64 h = mix64(key) & t.mask;
#pragma unroll 1
    for (u64 probe = 0; probe <= t.mask; ++probe) {
        Slot *s = &t.table[h];
        u64 k = __ldcg(&s->key);
        if (k == STBPE_EMPTY) {
            k = atomicCAS(&s->key, STBPE_EMPTY, key);
            if (k == STBPE_EMPTY) {
                if (atomicAdd(t.n_keys, 1ull) >= (t.mask + 1) / 4 * 3) atomicOr(t.error, 1u);
                k = key;
            }
        }
        if (k == key) {
            atomicAdd((u64 *)&s->count, n);
            return;
        }
        h = (h + 1) & t.mask;
        if ((probe & 63) == 63 && *(volatile unsigned int *)t.error) return;
    }
    atomicOr(t.error, 1u);
}

// key + 1 into a CTA's table, or false where no place is near
template <unsigned int SLOTS>
__device__ __forceinline__ bool rows_smem_add(u64 *s_key, int *s_val, u64 key) {
    unsigned int h = hash32(key) & (SLOTS - 1);
    bool done = false;
#pragma unroll 1
    for (int probe = 0; probe < 4 && !done; ++probe) {
        u64 x = lds_u64_volatile(&s_key[h]);
        if (x == STBPE_EMPTY) {
            x = atoms_cas_u64(&s_key[h], STBPE_EMPTY, key);
            if (x == STBPE_EMPTY) x = key;
        }
        if (x == key) {
            reds_add_s32(&s_val[h], 1);
            done = true;
        }
        h = (h + 1) & (SLOTS - 1);
    }
    return done;
}
__device__ __forceinline__ bool rows_byte_pair(u64 key) { return ((uint32_t)(key >> 32) | (uint32_t)key) < 256u; }
__device__ __forceinline__ unsigned int rows_byte_index(u64 key) { return ((uint32_t)(key >> 32) << 8) | (uint32_t)key; }

// Four cells (and the one behind them) of a flat batch, as one 16-byte and one 4-byte load
struct RowsQuad {
    int32_t w[5];
    unsigned int v[5];
    __device__ __forceinline__ void load(const int32_t *__restrict__ tokens, const uint8_t *__restrict__ valid, i64 q, i64 cells, bool aligned) {
#pragma unroll
        for (int k = 0; k < 5; ++k) w[k] = 0, v[k] = 0;
        if (aligned && q + 4 <= cells) {
            const int4 x = __ldg(reinterpret_cast<const int4 *>(tokens + q));
            const uchar4 y = __ldg(reinterpret_cast<const uchar4 *>(valid + q));
            w[0] = x.x, w[1] = x.y, w[2] = x.z, w[3] = x.w;
            v[0] = y.x, v[1] = y.y, v[2] = y.z, v[3] = y.w;
        } else {
            for (int k = 0; k < 4; ++k)
                if (q + k < cells) w[k] = tokens[q + k], v[k] = valid[q + k];
        }
        if ((threadIdx.x & 31) == 31 && q + 4 < cells) w[4] = tokens[q + 4], v[4] = valid[q + 4];
    }
    __device__ __forceinline__ void neighbour() {  // all lanes: the cell behind comes from the next lane
        const int32_t nw = __shfl_down_sync(0xFFFFFFFFu, w[0], 1);
        const unsigned int nv = __shfl_down_sync(0xFFFFFFFFu, v[0], 1);
        if ((threadIdx.x & 31) != 31) w[4] = nw, v[4] = nv;
    }
    // f(key) for every pair; `col` = column of the first cell.  A pair (i, i+1) of a row counts when both positions are valid
    // (gpu_tokenizer/utils.py:586).
    template <typename F>
    __device__ __forceinline__ void pairs(i64 col, i64 L, F &&f) const {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const bool last = ++col == L;  // the row ends here
            if (last) col = 0;
            if (!last && v[k] && v[k + 1]) f(((u64)(uint32_t)w[k] << 32) | (u64)(uint32_t)w[k + 1]);
            __syncwarp();
        }
    }
};

// Small batches: a CTA collects its pairs in shared memory and adds each distinct one once.
__global__ void __launch_bounds__(ROWS_SMALL_NT) rows_pairs_kernel(const int32_t *__restrict__ tokens, const uint8_t *__restrict__ valid, i64 B, i64 L,
                                                                   RowsTable t) {
    __shared__ u64 s_key[ROWS_SMALL_SLOTS];
    __shared__ int s_val[ROWS_SMALL_SLOTS];
    for (int i = threadIdx.x; i < ROWS_SMALL_SLOTS; i += ROWS_SMALL_NT) s_key[i] = STBPE_EMPTY, s_val[i] = 0;
    __syncthreads();
    const i64 cells = B * L;
    const bool aligned = (((uintptr_t)tokens & 15) | ((uintptr_t)valid & 3)) == 0;
    const i64 step = (i64)gridDim.x * ROWS_SMALL_NT * 4;
    i64 q = ((i64)blockIdx.x * ROWS_SMALL_NT + threadIdx.x) * 4;
    for (i64 q0 = (i64)blockIdx.x * ROWS_SMALL_NT * 4; q0 < cells; q0 += step, q += step) {  // uniform per CTA
        RowsQuad x;
        x.load(tokens, valid, q, cells, aligned);
        x.neighbour();
        x.pairs(q < cells ? q % L : 0, L, [&](u64 key) {
            if (!rows_smem_add<ROWS_SMALL_SLOTS>(s_key, s_val, key) && !(*(volatile unsigned int *)t.error)) rows_add(t, key, 1ull);
        });
    }
    __syncthreads();
    for (int k = threadIdx.x; k < ROWS_SMALL_SLOTS; k += ROWS_SMALL_NT) {  // each CTA from another place on
        const int i = (k + (int)blockIdx.x * (ROWS_SMALL_SLOTS / 128)) & (ROWS_SMALL_SLOTS - 1);
        if (s_val[i] && !(*(volatile unsigned int *)t.error)) rows_add(t, s_key[i], (u64)s_val[i]);
    }
}

// Up to 2^16 cells, a pair per thread straight into the table, equal pairs of a warp together: collecting them first costs a
// chain of trips to L2 for every entry that a thread adds afterwards (count of 16 x 512 cells of text 75 us, now 63, of 32 x 1024 cells
// with 32 736 pairs 212 and 174; 64 x 1024 cells of text 74 and 58).  Equal pairs queue up at their slot: 32 x 1024 equal cells took
// 91 us without the look at the warp, 50 with it as with tables; beyond 2^17 cells they are slower (255 x 1024: 64 and 50).
__global__ void __launch_bounds__(ROWS_SMALL_NT) rows_pairs_direct_kernel(const int32_t *__restrict__ tokens, const uint8_t *__restrict__ valid, i64 cells,
                                                                          i64 L, RowsTable t) {
    const i64 i = (i64)blockIdx.x * ROWS_SMALL_NT + threadIdx.x;
    const bool pair = i + 1 < cells && (i + 1) % L != 0 && valid[i] && valid[i + 1];
    const u64 key = pair ? ((u64)(uint32_t)tokens[i] << 32) | (u64)(uint32_t)tokens[i + 1] : STBPE_EMPTY;
    const unsigned int same = __match_any_sync(0xFFFFFFFFu, key);
    if (pair && (same & ((1u << (threadIdx.x & 31)) - 1u)) == 0u) rows_add(t, key, (u64)__popc(same));
}

// Large batches.  Bound by shared memory: a probe of the table costs two or three accesses that collide, an add to a directly
// indexed counter one, and early in a training nearly all pairs are of two bytes.  So a CTA whose first cells hold mostly
// such pairs (BYTES) counts them in 65 536 16-bit counters and the others in a smaller table beside them; else all go to one
// table of the whole room.  Every 15 turns of 4096 cells the counters are added to the batch's, so none overflows.
// (2048 x 4096 cells of mixed text: a count of 115 us with one table for all, now 60; 65 536 pairs of bytes 840 us for the call, now 230.)
struct RowsCells {
    const int32_t *__restrict__ tokens;
    const uint8_t *__restrict__ valid;
    i64 cells, L;
    bool aligned;
};
template <bool BYTES>
__device__ __forceinline__ void rows_count_large(const RowsCells &c, const RowsTable &t, unsigned char *smem) {
    constexpr unsigned int SLOTS = BYTES ? ROWS_MIXED_SLOTS : ROWS_LARGE_SLOTS;
    constexpr int TURNS = 65535 / (ROWS_LARGE_NT * 4);
    unsigned int *const s_count = reinterpret_cast<unsigned int *>(smem);  // two counters per word
    u64 *const s_key = reinterpret_cast<u64 *>(smem + (BYTES ? ROWS_BYTE_PAIRS * 2 : 0));
    int *const s_val = reinterpret_cast<int *>(s_key + SLOTS);
    if (BYTES)
        for (int i = threadIdx.x; i < ROWS_BYTE_PAIRS / 2; i += ROWS_LARGE_NT) s_count[i] = 0u;
    for (unsigned int i = threadIdx.x; i < SLOTS; i += ROWS_LARGE_NT) s_key[i] = STBPE_EMPTY, s_val[i] = 0;
    __syncthreads();
    // what a CTA has not collected itself
    auto add = [&](u64 key, u64 n) {
        if (*(volatile unsigned int *)t.error) return;
        if (!BYTES && rows_byte_pair(key))
            atomicAdd(t.bytes + rows_byte_index(key), n);
        else
            rows_add(t, key, n);
    };
    // (the counters of one first id are spread over the banks, those of neighbouring first ids shifted)
    auto flush_bytes = [&] {
        __syncthreads();
        for (unsigned int k = threadIdx.x; k < ROWS_BYTE_PAIRS / 2; k += ROWS_LARGE_NT) {
            const unsigned int i = (k + blockIdx.x * (ROWS_BYTE_PAIRS / 256)) & (ROWS_BYTE_PAIRS / 2 - 1);  // each CTA from another place on
            const unsigned int p = i ^ ((i >> 7) & 31u), x = s_count[p];
            if (!x) continue;
            s_count[p] = 0u;
            if (x & 0xFFFFu) atomicAdd(t.bytes + 2 * i, (u64)(x & 0xFFFFu));
            if (x >> 16) atomicAdd(t.bytes + 2 * i + 1, (u64)(x >> 16));
        }
        __syncthreads();
    };
    const i64 step = (i64)gridDim.x * ROWS_LARGE_NT * 4, col_step = step % c.L;
    i64 q = ((i64)blockIdx.x * ROWS_LARGE_NT + threadIdx.x) * 4, col = q % c.L;
    int turn = 0;
    for (i64 q0 = (i64)blockIdx.x * ROWS_LARGE_NT * 4; q0 < c.cells; q0 += step, q += step) {  // uniform per CTA
        RowsQuad x;
        x.load(c.tokens, c.valid, q, c.cells, c.aligned);
        if (BYTES && turn++ == TURNS) {
            flush_bytes();
            turn = 1;
        }
        x.neighbour();
        x.pairs(col, c.L, [&](u64 key) {
            if (BYTES && rows_byte_pair(key)) {
                const unsigned int i = rows_byte_index(key);
                reds_add_s32(reinterpret_cast<int *>(s_count + ((i >> 1) ^ ((i >> 8) & 31u))), (int)(1u << (16 * (i & 1u))));
            } else if (!rows_smem_add<SLOTS>(s_key, s_val, key)) {
                add(key, 1ull);
            }
        });
        col += col_step;
        if (col >= c.L) col -= c.L;
    }
    if (BYTES)
        flush_bytes();
    else
        __syncthreads();
    for (unsigned int k = threadIdx.x; k < SLOTS; k += ROWS_LARGE_NT) {
        const unsigned int i = (k + blockIdx.x * (SLOTS / 128)) & (SLOTS - 1);
        if (s_val[i]) add(s_key[i], (u64)s_val[i]);
    }
}
__global__ void __launch_bounds__(ROWS_LARGE_NT) rows_pairs_large_kernel(const int32_t *__restrict__ tokens, const uint8_t *__restrict__ valid, i64 B,
                                                                         i64 L, RowsTable t) {
    extern __shared__ __align__(16) unsigned char s_rows[];
    const RowsCells c = {tokens, valid, B * L, L, (((uintptr_t)tokens & 15) | ((uintptr_t)valid & 3)) == 0};
    const i64 q = ((i64)blockIdx.x * ROWS_LARGE_NT + threadIdx.x) * 4;
    RowsQuad x;
    x.load(tokens, valid, q, c.cells, c.aligned);
    x.neighbour();
    int balance = 0;
    x.pairs(q % L, L, [&](u64 key) { balance += rows_byte_pair(key) ? 1 : -1; });
    const int most = __syncthreads_count(balance > 0);
    if (2 * most > __syncthreads_count(balance != 0))
        rows_count_large<true>(c, t, s_rows);
    else
        rows_count_large<false>(c, t, s_rows);
}

// rank[i] += keys of the tile blockIdx.y that are smaller than key i
__global__ void __launch_bounds__(256) rows_rank_kernel(const u64 *__restrict__ keys, const u64 *n_keys, const unsigned int *error, unsigned int *rank) {
    __shared__ u64 s_k[ROWS_RANK_TILE];
    const i64 n = (i64)*n_keys;
    const i64 i = (i64)blockIdx.x * 256 + threadIdx.x, j0 = (i64)blockIdx.y * ROWS_RANK_TILE;
    if (*error || n > ROWS_RANK_MAX || (i64)blockIdx.x * 256 >= n || j0 >= n) return;
    const int m = (int)(n - j0 < ROWS_RANK_TILE ? n - j0 : ROWS_RANK_TILE);
    for (int k = threadIdx.x; k < ROWS_RANK_TILE; k += 256) s_k[k] = k < m ? keys[j0 + k] : STBPE_EMPTY;
    __syncthreads();
    if (i >= n) return;
    const u64 mine = keys[i];
    unsigned int r = 0;
#pragma unroll 8
    for (int k = 0; k < ((m + 7) & ~7); ++k) r += s_k[k] < mine ? 1u : 0u;
    if (r) atomicAdd(&rank[i], r);
}

// the histogram in ascending key order, unused rows -1 / 0, length (gpu_tokenizer/utils.py:622-635)
__global__ void rows_place_kernel(const u64 *__restrict__ keys, const i64 *__restrict__ counts, const unsigned int *__restrict__ rank, RowsTable t,
                                  int32_t *pair_keys, i64 *pair_counts, i64 cap, i64 *length) {
    const i64 n = (i64)*t.n_keys;
    if (*t.error || n > cap || n > ROWS_RANK_MAX) return;
    const i64 first = (i64)blockIdx.x * blockDim.x + threadIdx.x, step = (i64)gridDim.x * blockDim.x;
    for (i64 i = first; i < n; i += step) {
        const i64 at = rank[i];
        pair_keys[2 * at] = (int32_t)(keys[i] >> 32);
        pair_keys[2 * at + 1] = (int32_t)(keys[i] & 0xFFFFFFFFull);
        pair_counts[at] = counts[i];
    }
    for (i64 i = n + first; i < cap; i += step) {
        if (((uintptr_t)pair_keys & 7) == 0) {
            *reinterpret_cast<int2 *>(pair_keys + 2 * i) = make_int2(-1, -1);
        } else {
            pair_keys[2 * i] = -1;
            pair_keys[2 * i + 1] = -1;
        }
        pair_counts[i] = 0;
    }
    if (first == 0 && length) *length = n;
}

// best of n entries (per CTA): key, count, index into out[3 * blockIdx.x ...].  Entry i is keys[i * stride] and so on.  (One
// read-back of three words instead of three: four rounds of the seam on 16 x 512 cells 0.82 -> 0.79 ms.)
__global__ void __launch_bounds__(256) rows_best_kernel(const i64 *keys, const i64 *counts, const i64 *index, i64 stride, i64 n, i64 *out) {
    __shared__ i64 s_k[8], s_c[8], s_i[8];
    i64 bk = 0x7FFFFFFFFFFFFFFFll, bc = 0, bi = 0x7FFFFFFFFFFFFFFFll;
    auto take = [&](i64 k, i64 c, i64 i) {
        if (c > bc || (c == bc && (k < bk || (k == bk && i < bi)))) bk = k, bc = c, bi = i;
    };
    for (i64 i = (i64)blockIdx.x * 256 + threadIdx.x; i < n; i += (i64)gridDim.x * 256) take(keys[i * stride], counts[i * stride], index ? index[i * stride] : i);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        const i64 k = __shfl_down_sync(0xFFFFFFFFu, bk, d), c = __shfl_down_sync(0xFFFFFFFFu, bc, d), i = __shfl_down_sync(0xFFFFFFFFu, bi, d);
        take(k, c, i);
    }
    if ((threadIdx.x & 31) == 0) s_k[threadIdx.x >> 5] = bk, s_c[threadIdx.x >> 5] = bc, s_i[threadIdx.x >> 5] = bi;
    __syncthreads();
    if (threadIdx.x != 0) return;
    for (int w = 1; w < 8; ++w) take(s_k[w], s_c[w], s_i[w]);
    out[3 * blockIdx.x] = bk;
    out[3 * blockIdx.x + 1] = bc;
    out[3 * blockIdx.x + 2] = bi;
}

// One CTA per row, walking the row in chunks with a running output offset.  Writes never
// overtake reads (the output is a left compaction), so the row is rewritten in place.
//   mask[i] = tok[i]==a && tok[i+1]==b && valid[i] && valid[i+1]   on the pre-merge row
//   tok[i] = new where mask[i]; position i+1 is dropped where mask[i]   (utils.py:520-531)
//   stable compaction of the remaining valid positions, zero-filled tail (utils.py:347-410)
__global__ void __launch_bounds__(ROWS_NT)
    rows_merge_kernel(int32_t *tokens, uint8_t *valid, int32_t *lengths, i64 B, i64 L, int32_t a,
                      int32_t b, int32_t new_id, uint8_t *spans) {
    __shared__ int32_t s_tok[ROWS_CHUNK + 2];
    __shared__ uint8_t s_val[ROWS_CHUNK + 2];
    __shared__ int32_t s_out[ROWS_CHUNK];
    __shared__ int s_wcnt[ROWS_IPT * (ROWS_NT / 32)];
    __shared__ int s_total;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NW = ROWS_NT / 32;
    for (i64 row = blockIdx.x; row < B; row += gridDim.x) {
        int32_t *t = tokens + row * L;
        uint8_t *v = valid + row * L;
        uint8_t *sp = spans ? spans + row * (L - 1) : nullptr;
        i64 w = 0;  // output length so far (uniform across the CTA)
        int32_t carry_tok = 0;
        uint8_t carry_val = 0;  // pre-merge token / valid just before the chunk
        for (i64 base = 0; base < L; base += ROWS_CHUNK) {
            const int n = (int)((L - base) < ROWS_CHUNK ? (L - base) : ROWS_CHUNK);
            // s_tok[1 + i] = position base + i; s_tok[0] = carry; s_tok[n + 1] = lookahead
            for (int i = tid; i < n + 1; i += ROWS_NT) {
                const i64 p = base + i;
                s_tok[1 + i] = p < L ? t[p] : 0;
                s_val[1 + i] = p < L ? v[p] : 0;
            }
            if (tid == 0) {
                s_tok[0] = carry_tok;
                s_val[0] = base > 0 ? carry_val : 0;
            }
            __syncthreads();
            int32_t outv[ROWS_IPT];
            unsigned int surv = 0;
#pragma unroll
            for (int j = 0; j < ROWS_IPT; ++j) {
                const int i = j * ROWS_NT + tid;
                outv[j] = 0;
                if (i < n) {
                    const int32_t tm1 = s_tok[i], t0 = s_tok[i + 1], t1 = s_tok[i + 2];
                    const bool vm1 = s_val[i], v0 = s_val[i + 1], v1 = s_val[i + 2];
                    const bool M0 = t0 == a && t1 == b && v0 && v1 && (base + i + 1 < L);
                    const bool D0 = tm1 == a && t0 == b && vm1 && v0;
                    if (sp && base + i < L - 1) sp[base + i] = (uint8_t)M0;
                    outv[j] = M0 ? new_id : t0;
                    if (v0 && !D0) surv |= 1u << j;
                }
            }
            const int32_t next_carry_tok = s_tok[n];
            const uint8_t next_carry_val = s_val[n];
            unsigned int bal[ROWS_IPT];
#pragma unroll
            for (int j = 0; j < ROWS_IPT; ++j) {
                bal[j] = __ballot_sync(0xFFFFFFFFu, (surv >> j) & 1u);
                if (lane == 0) s_wcnt[j * NW + warp] = __popc(bal[j]);
            }
            __syncthreads();
            if (warp == 0) {
                // exclusive scan of IPT*NW (=64) counts, 2 per lane
                int v0c = s_wcnt[lane * 2], v1c = s_wcnt[lane * 2 + 1];
                int sum = v0c + v1c, incl = sum;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    int o = __shfl_up_sync(0xFFFFFFFFu, incl, d);
                    if (lane >= d) incl += o;
                }
                s_wcnt[lane * 2] = incl - sum;
                s_wcnt[lane * 2 + 1] = incl - sum + v0c;
                if (lane == 31) s_total = incl;
            }
            __syncthreads();
            const unsigned int lt = (1u << lane) - 1u;
#pragma unroll
            for (int j = 0; j < ROWS_IPT; ++j)
                if ((surv >> j) & 1u) s_out[s_wcnt[j * NW + warp] + __popc(bal[j] & lt)] = outv[j];
            __syncthreads();
            const int produced = s_total;
            for (int i = tid; i < produced; i += ROWS_NT) {
                t[w + i] = s_out[i];
                v[w + i] = 1;
            }
            w += produced;
            carry_tok = next_carry_tok;
            carry_val = next_carry_val;
            __syncthreads();
        }
        for (i64 i = w + tid; i < L; i += ROWS_NT) {
            t[i] = 0;
            v[i] = 0;
        }
        if (tid == 0 && lengths) lengths[row] = (int32_t)w;
        __syncthreads();
    }
}

thread_local std::string g_rows_err;

}  // namespace

#define RCK(call)                                                        \
    do {                                                                 \
        cudaError_t c_ = (call);                                         \
        if (c_ != cudaSuccess) {                                         \
            g_rows_err = std::string(#call) + ": " + cudaGetErrorString(c_); \
            cudaGetLastError();                                          \
            return STBPE_E_CUDA;                                         \
        }                                                                \
    } while (0)

extern "C" {

STBPE_VISIBLE int stbpe_rows_count_pairs(const int32_t *tokens, const uint8_t *valid, int64_t B, int64_t L,
                                         int32_t *pair_keys, int64_t *pair_counts, int64_t cap,
                                         int64_t *length_dev, void *stream) {
    cudaStream_t s = (cudaStream_t)stream;
    if (B < 0 || L < 0 || cap < 0) return STBPE_E_BADARG;
    const i64 total = (B > 0 && L > 1) ? B * (L - 1) : 0;
    int dev = 0;
    RCK(cudaGetDevice(&dev));
    // A batch of text holds a few thousand distinct pairs among millions of positions, so the table starts at 2^16
    // slots (1 MB, cleared and scanned in microseconds; for twice the positions it was 512 MB on a batch of
    // 2048 x 4096) and the count is repeated with sixteen times the slots when the pairs do not fit.
    u64 largest = 1024;
    while (largest < (u64)total * 2 && largest < (1ull << 28)) largest <<= 1;
    u64 slots = largest < (1u << 16) ? largest : (1u << 16);
    stbpe::Block pin;
    RCK(stbpe::pinned_blocks().get(0, 4096, &pin));
    volatile u64 *got = (volatile u64 *)pin.p;
    int rc = STBPE_OK;
    const bool large = B * L >= ROWS_LARGE_CELLS;
    for (;;) {
        const u64 room = slots + (large ? ROWS_BYTE_PAIRS : 0), most = room < (u64)(total > 0 ? total : 1) ? room : (u64)(total > 0 ? total : 1);
        const size_t keys_at = slots * sizeof(Slot), counts_at = keys_at + most * 8, rank_at = counts_at + most * 8,
                     meta_at = (rank_at + most * 4 + 255) & ~(size_t)255, bytes_at = meta_at + 256;
        stbpe::Block b;
        cudaError_t c = stbpe::device_blocks().get(dev, bytes_at + (large ? ROWS_BYTE_PAIRS * sizeof(u64) : 0), &b);
        if (c == cudaSuccess) {
            unsigned char *base = (unsigned char *)b.p;
            RowsTable t;
            t.table = (Slot *)base;
            t.mask = slots - 1;
            t.n_keys = (u64 *)(base + meta_at);
            t.error = (unsigned int *)(t.n_keys + 1);
            t.bytes = large ? (u64 *)(base + bytes_at) : nullptr;
            u64 *n_out = t.n_keys + 2;
            u64 *keys = (u64 *)(base + keys_at);
            i64 *counts = (i64 *)(base + counts_at);
            unsigned int *rank = (unsigned int *)(base + rank_at);
            const i64 quads = (B * L + 3) / 4;
            const i64 ranked = (i64)most < ROWS_RANK_MAX ? (i64)most : ROWS_RANK_MAX;  // more pairs than these take the radix sort
            const int nt = large ? ROWS_LARGE_NT : ROWS_SMALL_NT;
            const i64 want = (quads + nt - 1) / nt, most_ctas = large ? 148 : 148 * 4;
            const unsigned int grid = (unsigned int)(want < most_ctas ? want : most_ctas);
            rows_init_kernel<<<slots < (1u << 18) ? 64 : 592, 256, 0, s>>>(t, rank, (unsigned int)(most < ROWS_RANK_MAX ? most : ROWS_RANK_MAX));
            if (total > 0 && large) {
                cudaFuncSetAttribute(rows_pairs_large_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ROWS_LARGE_SMEM);
                rows_pairs_large_kernel<<<grid, ROWS_LARGE_NT, ROWS_LARGE_SMEM, s>>>(tokens, valid, B, L, t);
            } else if (total > 0 && B * L <= ROWS_DIRECT_CELLS) {
                rows_pairs_direct_kernel<<<(unsigned int)((B * L + ROWS_SMALL_NT - 1) / ROWS_SMALL_NT), ROWS_SMALL_NT, 0, s>>>(tokens, valid, B * L, L, t);
            } else if (total > 0) {
                rows_pairs_kernel<<<grid, ROWS_SMALL_NT, 0, s>>>(tokens, valid, B, L, t);
            }
            if (total > 0) rows_export_kernel<<<slots < (1u << 18) ? 64 : 592, 256, 0, s>>>(t, keys, counts, n_out, (i64)most);
            if (total > 0) rows_rank_kernel<<<dim3((unsigned int)((ranked + 255) / 256), (unsigned int)((ranked + ROWS_RANK_TILE - 1) / ROWS_RANK_TILE)), 256, 0, s>>>(keys, t.n_keys, t.error, rank);
            i64 wb = (cap + 255) / 256;
            if (wb > 148 * 16) wb = 148 * 16;
            rows_place_kernel<<<(unsigned int)(wb > 0 ? wb : 1), 256, 0, s>>>(keys, counts, rank, t, pair_keys, (i64 *)pair_counts, cap, (i64 *)length_dev);
            c = cudaGetLastError();
            if (c == cudaSuccess) c = cudaMemcpyAsync(pin.p, t.n_keys, 2 * sizeof(u64), cudaMemcpyDeviceToHost, s);
            if (c == cudaSuccess) c = cudaStreamSynchronize(s);
            if (c == cudaSuccess) {
                const i64 n = (i64)got[0];
                const bool full = (got[1] & 0xFFFFFFFFull) != 0;
                if (full && slots < largest) {
                    stbpe::device_blocks().put(dev, b);
                    slots = slots * 16 < largest ? slots * 16 : largest;
                    continue;
                }
                if (full || n > cap) {
                    rc = STBPE_E_CAPACITY;  // "pair workspace capacity exceeded" (utils.py:619-620)
                } else if (n > ROWS_RANK_MAX) {
                    // many pairs: radix sort
                    size_t tmp = 0;
                    cub::DeviceRadixSort::SortPairs(nullptr, tmp, keys, keys, counts, counts, (int)n, 0, 64, s);
                    stbpe::Block w;
                    const size_t side = ((size_t)n * 8 + 255) & ~(size_t)255;
                    c = stbpe::device_blocks().get(dev, 2 * side + tmp + 256, &w);
                    if (c == cudaSuccess) {
                        u64 *sk = (u64 *)w.p;
                        i64 *sc = (i64 *)((unsigned char *)w.p + side);
                        cub::DeviceRadixSort::SortPairs((unsigned char *)w.p + 2 * side, tmp, keys, sk, counts, sc, (int)n, 0, 64, s);
                        rows_write_kernel<<<(unsigned int)(wb > 0 ? wb : 1), 256, 0, s>>>(sk, sc, n, pair_keys, (i64 *)pair_counts, cap, (i64 *)length_dev);
                        c = cudaGetLastError();
                        if (c == cudaSuccess) c = cudaStreamSynchronize(s);
                        if (c == cudaSuccess) stbpe::device_blocks().put(dev, w);
                    }
                }
            }
        }
        if (c != cudaSuccess) {  // the blocks may still be in use: they are not handed on
            g_rows_err = cudaGetErrorString(c);
            cudaGetLastError();
            return STBPE_E_CUDA;
        }
        stbpe::device_blocks().put(dev, b);
        break;
    }
    stbpe::pinned_blocks().put(0, pin);
    return rc;
}

// Best entry of a histogram: maximum count, ties to the smallest key (gpu_tokenizer/trainers/bpe_gpu.py:106-127).
STBPE_VISIBLE int stbpe_select_pair(const int64_t *keys, const int64_t *counts, int64_t n, int64_t *key, int64_t *count, int64_t *index,
                                    void *stream) {
    cudaStream_t s = (cudaStream_t)stream;
    if (n < 0 || !key || !count || !index || (n > 0 && (!keys || !counts))) return STBPE_E_BADARG;
    *key = 0, *count = 0, *index = -1;
    if (n == 0) return STBPE_OK;
    int dev = 0;
    RCK(cudaGetDevice(&dev));
    stbpe::Block b, pin;
    RCK(stbpe::device_blocks().get(dev, 65536, &b));
    RCK(stbpe::pinned_blocks().get(0, 4096, &pin));
    const i64 want = (n + 1023) / 1024;
    const int grid = (int)(want < 148 ? want : 148);
    rows_best_kernel<<<grid, 256, 0, s>>>((const i64 *)keys, (const i64 *)counts, nullptr, 1, n, (i64 *)b.p);
    if (grid > 1) rows_best_kernel<<<1, 256, 0, s>>>((const i64 *)b.p, (const i64 *)b.p + 1, (const i64 *)b.p + 2, 3, grid, (i64 *)b.p + 3 * 256);
    RCK(cudaGetLastError());
    i64 *h = (i64 *)pin.p;
    RCK(cudaMemcpyAsync(h, (i64 *)b.p + (grid > 1 ? 3 * 256 : 0), 3 * sizeof(i64), cudaMemcpyDeviceToHost, s));
    RCK(cudaStreamSynchronize(s));
    if (h[1] > 0) *key = h[0], *count = h[1], *index = h[2];
    stbpe::device_blocks().put(dev, b);
    stbpe::pinned_blocks().put(0, pin);
    return STBPE_OK;
}

STBPE_VISIBLE int stbpe_rows_apply_merge(int32_t *tokens, uint8_t *valid, int32_t *lengths, int64_t B,
                                         int64_t L, int32_t a, int32_t b, int32_t new_id, uint8_t *spans,
                                         void *stream) {
    cudaStream_t s = (cudaStream_t)stream;
    if (B < 0 || L < 0) return STBPE_E_BADARG;
    if (B == 0 || L == 0) return STBPE_OK;
    i64 grid = B < 148 * 8 ? B : 148 * 8;
    rows_merge_kernel<<<(unsigned int)grid, ROWS_NT, 0, s>>>(tokens, valid, lengths, B, L, a, b, new_id, spans);
    RCK(cudaGetLastError());
    return STBPE_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------------------
// Pair counting for callers that must not allocate.
//
// stbpe_rows_count_pairs above takes its hash table, staging arrays and sort workspace from the
// process-wide block cache, which allocates when it holds nothing that fits.  Two kinds of caller of this library cannot
// afford that.  The reference's trainer sizes its batches to fill device memory (its
// --target-util flag) and hands every byte to preallocated workspaces before the merge loop
// starts, so an allocation made in the middle of the loop is the one that fails; and it
// overlaps copies and kernels on three streams per device, which a cudaMalloc / cudaFree
// stalls, because those calls synchronise the whole device.
//
// This variant works out of one fixed scratch block that is part of the library image: a
// file-scope __device__ array.  Every GPU on which the library is loaded holds the block
// (STBPE_STATIC_SCRATCH_BYTES, about 5.3 MB) from load to exit.  In host code the array's
// name is only a handle for the runtime, not a device address, so the entry point asks
// cudaGetSymbolAddress for the address once per device, with that device current, and hands
// the returned pointer to the kernels.  That look-up happens inside the first call made on
// each device; make that first call outside any stream capture.
//
// All calls share the block and it keeps what the last call left there: the table and the
// counters are cleared at the start of every call, and two calls that overlap on the GPU
// (different streams, or different host threads) race on it -- serialise them.
// ---------------------------------------------------------------------------------------
#define STBPE_STATIC_MAX_POSITIONS (1 << 16)  /* largest B*(L-1) accepted */
#define STBPE_STATIC_TABLE_SLOTS (1 << 17)
#define STBPE_STATIC_SORT_BYTES (1 << 20)
#define STBPE_STATIC_SCRATCH_BYTES                                                              \
    ((size_t)STBPE_STATIC_TABLE_SLOTS * sizeof(Slot) + (size_t)4 * STBPE_STATIC_MAX_POSITIONS * 8 + \
     256 + (size_t)STBPE_STATIC_SORT_BYTES)

static __device__ __align__(256) unsigned char g_static_scratch[STBPE_STATIC_SCRATCH_BYTES];

namespace {
std::mutex g_static_mu;
unsigned char *g_static_ptr[64] = {};

// device address of the scratch block on the current device (looked up once per device)
int static_scratch(unsigned char **out, char *err, size_t err_len) {
    int dev = -1;
    cudaError_t c = cudaGetDevice(&dev);
    if (c != cudaSuccess || dev < 0 || dev >= 64) {
        if (err) snprintf(err, err_len, "cudaGetDevice failed or device ordinal out of range: %s", cudaGetErrorString(c));
        return STBPE_E_CUDA;
    }
    std::lock_guard<std::mutex> lock(g_static_mu);
    if (g_static_ptr[dev]) {
        // a cudaDeviceReset since the look-up gives the block a new address: ask again if the cached
        // one is no longer device memory of this device (a query, no allocation)
        cudaPointerAttributes at;
        if (cudaPointerGetAttributes(&at, g_static_ptr[dev]) != cudaSuccess || at.type != cudaMemoryTypeDevice ||
            at.device != dev) {
            cudaGetLastError();
            g_static_ptr[dev] = nullptr;
        }
    }
    if (!g_static_ptr[dev]) {
        void *p = nullptr;
        c = cudaGetSymbolAddress(&p, g_static_scratch);
        if (c != cudaSuccess || !p) {
            if (err) snprintf(err, err_len, "cudaGetSymbolAddress(scratch) failed: %s", cudaGetErrorString(c));
            cudaGetLastError();
            return STBPE_E_CUDA;
        }
        g_static_ptr[dev] = static_cast<unsigned char *>(p);
    }
    *out = g_static_ptr[dev];
    return STBPE_OK;
}
}  // namespace

#define SCK(call)                                                                         \
    do {                                                                                  \
        cudaError_t c_ = (call);                                                          \
        if (c_ != cudaSuccess) {                                                          \
            if (err) snprintf(err, err_len, "%s: %s", #call, cudaGetErrorString(c_));     \
            cudaGetLastError();                                                           \
            return STBPE_E_CUDA;                                                          \
        }                                                                                 \
    } while (0)

extern "C" STBPE_VISIBLE int stbpe_rows_count_pairs_noalloc(const int32_t *tokens, const uint8_t *valid,
                                                            int64_t B, int64_t L, int32_t *pair_keys,
                                                            int64_t *pair_counts, int64_t cap,
                                                            int64_t *length_dev, void *stream, char *err,
                                                            size_t err_len) {
    cudaStream_t s = (cudaStream_t)stream;
    if (err && err_len) err[0] = 0;
    if (B < 0 || L < 0 || cap < 0) {
        if (err) snprintf(err, err_len, "negative size");
        return STBPE_E_BADARG;
    }
    const i64 total = (B > 0 && L > 1) ? B * (L - 1) : 0;
    if (total > STBPE_STATIC_MAX_POSITIONS) {
        if (err)
            snprintf(err, err_len,
                     "batch too large for the fixed scratch block: B*(L-1) = %lld pair positions, limit %d "
                     "(use stbpe_rows_count_pairs, which allocates)",
                     (long long)total, STBPE_STATIC_MAX_POSITIONS);
        return STBPE_E_CAPACITY;
    }
    unsigned char *base = nullptr;
    int rc = static_scratch(&base, err, err_len);
    if (rc != STBPE_OK) return rc;
    // carve the block: table | keys | counts | sorted keys | sorted counts | counters | sort workspace
    Slot *table = reinterpret_cast<Slot *>(base);
    u64 *keys = reinterpret_cast<u64 *>(base + (size_t)STBPE_STATIC_TABLE_SLOTS * sizeof(Slot));
    i64 *counts = reinterpret_cast<i64 *>(keys + STBPE_STATIC_MAX_POSITIONS);
    u64 *skeys = reinterpret_cast<u64 *>(counts + STBPE_STATIC_MAX_POSITIONS);
    i64 *scounts = reinterpret_cast<i64 *>(skeys + STBPE_STATIC_MAX_POSITIONS);
    u64 *meta = reinterpret_cast<u64 *>(scounts + STBPE_STATIC_MAX_POSITIONS);
    void *sort_ws = reinterpret_cast<unsigned char *>(meta) + 256;
    const u64 *sorted_keys = skeys;
    const i64 *sorted_counts = scounts;
    i64 n = 0;
    if (total > 0) {
        RowsTable t;
        t.table = table;
        t.mask = STBPE_STATIC_TABLE_SLOTS - 1;
        t.n_keys = meta;
        t.error = reinterpret_cast<unsigned int *>(meta + 1);
        t.bytes = nullptr;
        // the block still holds the previous call's table and counters: start from zero
        SCK(cudaMemsetAsync(meta, 0, 256, s));
        rows_clear_kernel<<<256, 256, 0, s>>>(t);
        i64 blocks = (total + 255) / 256;
        rows_count_kernel<<<(unsigned int)blocks, 256, 0, s>>>(tokens, valid, B, L, t);
        SCK(cudaGetLastError());
        u64 hmeta[2] = {0, 0};
        SCK(cudaMemcpyAsync(hmeta, meta, sizeof(hmeta), cudaMemcpyDeviceToHost, s));
        SCK(cudaStreamSynchronize(s));
        n = (i64)hmeta[0];
        if ((hmeta[1] & 0xFFFFFFFFull) != 0 || n > cap) {
            if (err) snprintf(err, err_len, "pair workspace capacity exceeded (%lld unique pairs, cap %lld)", (long long)n, (long long)cap);
            return STBPE_E_CAPACITY;
        }
        if (n > 0) {
            // Sort through double buffers: the two key arrays and the two count arrays of the block are
            // the sort's ping-pong buffers, so its own workspace holds only digit counters (without
            // them it would ask for a second copy of keys and counts, 1 MiB at the size limit).  The
            // workspace size is checked before anything else is queued on the shared block.
            cub::DoubleBuffer<u64> dk(keys, skeys);
            cub::DoubleBuffer<i64> dc(counts, scounts);
            size_t need = 0;
            cub::DeviceRadixSort::SortPairs(nullptr, need, dk, dc, (int)n, 0, 64, s);
            if (need > (size_t)STBPE_STATIC_SORT_BYTES) {
                if (err) snprintf(err, err_len, "sort workspace of %zu bytes exceeds the reserved %d", need, STBPE_STATIC_SORT_BYTES);
                return STBPE_E_CAPACITY;
            }
            SCK(cudaMemsetAsync(meta, 0, sizeof(u64), s));
            rows_export_kernel<<<256, 256, 0, s>>>(t, keys, counts, meta, n);
            cub::DeviceRadixSort::SortPairs(sort_ws, need, dk, dc, (int)n, 0, 64, s);
            SCK(cudaGetLastError());
            sorted_keys = dk.Current();
            sorted_counts = dc.Current();
        }
    }
    if (cap > 0) {
        i64 blocks = (cap + 255) / 256;
        if (blocks > 148 * 32) blocks = 148 * 32;
        rows_write_kernel<<<(unsigned int)blocks, 256, 0, s>>>(sorted_keys, sorted_counts, n, pair_keys, (i64 *)pair_counts, cap, (i64 *)length_dev);
        SCK(cudaGetLastError());
    } else if (length_dev) {
        SCK(cudaMemsetAsync(length_dev, 0, sizeof(i64), s));
    }
    SCK(cudaStreamSynchronize(s));
    return STBPE_OK;
}
