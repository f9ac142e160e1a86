// K2, wide path: first count of a fresh stream whose ids are all below 65 536 (a 16-bit vocabulary).
//
// The pair space is 2^32 keys and a Zipf-like id stream touches 10^8 of them, so a histogram kept in
// one place is bound by random memory accesses, not by the stream (one scattered reduction per token
// into a table in HBM ran at 37 G sector requests per second, 4 % of the stream rate).  Random
// reductions are six times faster while their target stays in L2 (measured on B200: 227 G per second
// into 64 MB, 21 G per second into 4 GB), so the count is split in two passes that never touch HBM at
// random:
//
//   pass 1  partition_pairs_kernel reads the stream once.  Pairs of two ids below 256 (44 % of a
//           Zipf(1.1) stream) go to 16-bit shared-memory counters as in the byte-level kernel.  Every
//           other pair becomes one 32-bit word, mix32((a << 16) | b), and is appended to the
//           partition named by the word's top 8 bits: per CTA a ring of 64 words per partition in
//           shared memory, flushed with coalesced stores after every batch of tokens into a region
//           of the partition that belongs to this CTA alone (no reservation, hence no atomic and no
//           round trip to memory in the loop; with one global cursor per partition the flush waited
//           for 256 dependent reservations per batch and the pass took 13.4 ms instead of 4).  The
//           mix is a bijection, so partitions are balanced whatever the ids, and the word still
//           identifies the pair.
//   pass 2  sub_partition_kernel orders the words of every piece of a region by their next bits.
//   pass 3  build_table_kernel: the slot index of a key starts with the same bits as its word, so a CTA that
//           takes a range of words owns a range of slots.  It counts the words in shared memory and
//           writes the slots out, occupied or not: the table is not cleared before and no atomic reaches L2.
//           200 M ids, 31 M pairs: 1.2 ms for both passes (6.2 ms when every word was added to the table with
//           one or two atomics in L2, a partition at a time).
// Several ranks: the owner of a partition adds its words out of every rank's regions
// (partition_table_peers_kernel); the table slice that a launch touches stays in L2.  One rank does the same with a long
// stream into a table of 2^29 slots or more (wide_one_by_one in engine.cu has the measurements).
//
// An id of 65 536 or more, or a partition region that outgrows its buffer, raises
// STBPE_DERR_DENSE_OVERFLOW and the host recounts with the general kernel.
#pragma once
#include "stream.cuh"

#define STBPE_PART_RING 64          // words per partition and CTA between two flushes
#define STBPE_PART_THREADS 1024
#define STBPE_PART_UNROLL 3         // uint4 loads per thread and batch: 12 288 tokens per CTA batch
static_assert(STBPE_PARTS == 8 * (STBPE_PART_THREADS / 32), "a warp of the first pass serves eight rings");
#define STBPE_PART_CACHE_BITS 12    // log2 of the entries of the per-CTA word cache of partition_table_peers_kernel (32 KB)
#define STBPE_PART_CACHE (1 << STBPE_PART_CACHE_BITS)
#define STBPE_PART_SHIFT (32 - STBPE_PART_BITS)
#define STBPE_PART_SMEM_BYTES (32768 * 4 + STBPE_PARTS * STBPE_PART_RING * 4 + 2 * STBPE_PARTS * 4)

struct PartBuffers {
    uint32_t *words;        // [partition][CTA of pass 1] regions of `cap` words
    unsigned int *fill;     // words in each region
    i64 cap;
    int n_cta;              // grid size of pass 1
};

// Several ranks: every rank partitions its own rows, then the owner of a partition (partition modulo
// the number of ranks) counts the partition's words out of every rank's regions with plain peer
// loads over NVLink, and sums the ranks' counters of the hot pairs it owns.  The buffers of a rank
// live in one allocation that its peers map: a header {cap, n_cta}, the region fills, the 65 536 hot
// counters, the regions.
#define STBPE_WIDE_HEADER_BYTES 256
struct WideHeader {
    i64 cap;
    int n_cta;
};
struct WidePeers {
    const unsigned char *block[STBPE_MAX_PEERS];  // every rank's allocation ([rank] = own)
    int world, rank;
};
__host__ __device__ __forceinline__ size_t wide_fill_bytes(int n_cta) {
    return (((size_t)STBPE_PARTS * n_cta * sizeof(unsigned int)) + 255) & ~(size_t)255;
}
__host__ __device__ __forceinline__ const unsigned int *wide_fill(const unsigned char *block) {
    return reinterpret_cast<const unsigned int *>(block + STBPE_WIDE_HEADER_BYTES);
}
__host__ __device__ __forceinline__ const u64 *wide_dense(const unsigned char *block, int n_cta) {
    return reinterpret_cast<const u64 *>(block + STBPE_WIDE_HEADER_BYTES + wide_fill_bytes(n_cta));
}
__host__ __device__ __forceinline__ const uint32_t *wide_words(const unsigned char *block, int n_cta) {
    return reinterpret_cast<const uint32_t *>(block + STBPE_WIDE_HEADER_BYTES + wide_fill_bytes(n_cta) +
                                              65536 * sizeof(u64));
}

__device__ __forceinline__ void part_append(const PartBuffers &pb, unsigned int *s_ring, unsigned int *s_cur,
                                            unsigned int *s_fill, unsigned int *derr, uint32_t word) {
    const unsigned int p = word >> STBPE_PART_SHIFT;
    const unsigned int pos = atomicAdd(&s_cur[p], 1u);
    if (pos < STBPE_PART_RING) {
        // rings fill at about the same pace, so slot `pos` of every ring would sit in the same bank:
        // rotate each ring by its partition number
        s_ring[p * STBPE_PART_RING + ((pos + p) & (STBPE_PART_RING - 1))] = word;
    } else {  // ring full before the flush (far out in the tail of the batch statistics): append directly
        const unsigned int g = atomicAdd(&s_fill[p], 1u);
        if ((i64)g < pb.cap)
            pb.words[((i64)p * pb.n_cta + blockIdx.x) * pb.cap + g] = word;
        else
            atomicOr(derr, STBPE_DERR_DENSE_OVERFLOW);
    }
}

__device__ __forceinline__ void part_pair(const PartBuffers &pb, unsigned int *s_tab, unsigned int *s_ring,
                                          unsigned int *s_cur, unsigned int *s_fill, u64 *g_dense,
                                          unsigned int *derr, uint32_t t0, uint32_t t1) {
    // the classes are worked out first and the two kinds of add follow one another, so that the lanes
    // of a warp, whose pairs fall into different classes, share the instructions of each kind
    const uint32_t both = t0 | t1;             // bit 31 set: the right token starts a row or lies past the end
    const bool hot = both < 256u;
    const bool wide = !hot && both < 65536u;
    if (hot) dense_add(s_tab, g_dense, derr, t0, t1);
    if (wide) part_append(pb, s_ring, s_cur, s_fill, derr, mix32((t0 << 16) | t1));
    if (!hot && !wide && !(t1 & STBPE_FLAG)) atomicOr(derr, STBPE_DERR_DENSE_OVERFLOW);
}

template <typename T>
__global__ void __launch_bounds__(STBPE_PART_THREADS, 1)
    partition_pairs_kernel(EngineDev e, u64 *g_dense, PartBuffers pb) {
    constexpr int UNROLL = sizeof(T) == 2 ? 2 : STBPE_PART_UNROLL;  // a unit is eight or four tokens
    extern __shared__ __align__(16) unsigned int s_all[];
    unsigned int *s_tab = s_all;                                  // 32 768 words of 16-bit counters
    unsigned int *s_ring = s_all + 32768;                         // STBPE_PARTS rings
    unsigned int *s_cur = s_ring + STBPE_PARTS * STBPE_PART_RING;  // ring fill
    unsigned int *s_fill = s_cur + STBPE_PARTS;                   // words this CTA has stored per partition
    for (int i = threadIdx.x; i < 32768; i += STBPE_PART_THREADS) s_tab[i] = 0u;
    for (int i = threadIdx.x; i < STBPE_PARTS; i += STBPE_PART_THREADS) s_cur[i] = s_fill[i] = 0u;
    __syncthreads();
    const uint4 *units = reinterpret_cast<const uint4 *>(e.tiles);
    const i64 n_units = (i64)e.n_tiles * (STBPE_TILE * sizeof(T) / 16);
    unsigned int *derr = &e.st->error;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint4 v[UNROLL];
    uint32_t nx[UNROLL];
    // the loads of a batch are issued before the flush of the batch before it, so that their trip to
    // memory runs under the flush and its two CTA barriers
    const i64 step = (i64)gridDim.x * STBPE_PART_THREADS * UNROLL;
    i64 base = (i64)blockIdx.x * STBPE_PART_THREADS * UNROLL;
    if (base < n_units) load_unit_batch<T, UNROLL, STBPE_PART_THREADS>(units, base, n_units, v, nx);
    for (; base < n_units; base += step) {
#pragma unroll
        for (int u = 0; u < UNROLL; ++u)
            unit_pairs<T>(v[u], nx[u], [&](uint32_t t0, uint32_t t1) {
                if (sizeof(T) == 2) t1 = (t1 & 0x7FFFu) | ((t1 & 0x8000u) << 16);
                part_pair(pb, s_tab, s_ring, s_cur, s_fill, g_dense, derr, t0 & Tok<T>::IDMASK, t1);
            });
        if (base + step < n_units) load_unit_batch<T, UNROLL, STBPE_PART_THREADS>(units, base + step, n_units, v, nx);
        __syncthreads();
        // flush into this CTA's regions: a warp serves its eight rings four at a time, eight lanes per ring, 32
        // consecutive bytes a turn, which start where the region has got to (eight rings at once, four lanes each, took as many
        // turns of 16 bytes: the pass over 200 M ids 0.75 ms, now 0.68; one ring at a time cost eight times the bookkeeping)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int p = warp * (STBPE_PARTS / (STBPE_PART_THREADS / 32)) + half * 4 + (lane >> 3);
            const unsigned int n = min(s_cur[p], (unsigned int)STBPE_PART_RING);
            const unsigned int g = s_fill[p];
            __syncwarp();
            if ((i64)g + n <= pb.cap) {
                uint32_t *dst = pb.words + ((i64)p * pb.n_cta + blockIdx.x) * pb.cap + g;
                for (unsigned int k = lane & 7; k < n; k += 8)
                    dst[k] = s_ring[p * STBPE_PART_RING + ((k + p) & (STBPE_PART_RING - 1))];
            } else if ((lane & 7) == 0) {
                atomicOr(derr, STBPE_DERR_DENSE_OVERFLOW);
            }
            if ((lane & 7) == 0) {
                s_fill[p] = g + n;
                s_cur[p] = 0u;
            }
        }
        __syncthreads();
    }
    for (int p = threadIdx.x; p < STBPE_PARTS; p += STBPE_PART_THREADS) {
        const unsigned int n = s_fill[p];
        pb.fill[(i64)p * pb.n_cta + blockIdx.x] = (i64)n < pb.cap ? n : (unsigned int)pb.cap;
    }
    for (int p = threadIdx.x; p < 32768; p += STBPE_PART_THREADS) {
        const unsigned int x = s_tab[p];
        const unsigned int w = (unsigned int)p ^ (((unsigned int)p >> 7) & 31u);  // inverse of dense_word
        if (x & 0xFFFFu) atomicAdd(&g_dense[2 * w], (u64)(x & 0xFFFFu));
        if (x >> 16) atomicAdd(&g_dense[2 * w + 1], (u64)(x >> 16));
    }
}

// Add n occurrences of a key to the pair table during the first count: no maxima to keep (a full
// refresh follows), and a key that is already there costs one load and one reduction without result.
__device__ __forceinline__ bool table_count_n(const EngineDev &e, u64 key, u64 h, u64 n, unsigned int &fresh) {
    for (unsigned int probe = 0; probe_on(e, probe); ++probe) {
        Slot *s = &e.table[h];
        u64 k = __ldcg(&s->key);
        if (k == STBPE_EMPTY) {
            const u64 old = atomicCAS(&s->key, STBPE_EMPTY, key);
            if (old == STBPE_EMPTY) {
                ++fresh;
                k = key;
            } else {
                k = old;
            }
        }
        if (k == key) {
            atomicAdd((u64 *)&s->count, n);  // result unused: a reduction
            return true;
        }
        h = (h + 1) & e.mask;
    }
    atomicOr(&e.st->error, STBPE_DERR_TABLE_FULL);
    return false;
}

__device__ __forceinline__ void part_word_to_table(const EngineDev &e, uint32_t x, u64 n, unsigned int &fresh) {
    const uint32_t ab = unmix32(x);
    const u64 key = ((u64)(ab >> 16) << 32) | (u64)(ab & 0xFFFFu);
    table_count_n(e, key, slot_of_word(e, x), n, fresh);
}

// pass 2, one rank: the words of every chunk (a piece of a pass-1 region of at most CHUNK words) in
// order of their next `sub_bits` bits, in place; offs[chunk][d] = where the words of digit d start.
// One returning shared-memory atomic per word gives its rank inside its digit, the words wait in registers
// meanwhile and go back through shared memory in order.
#define STBPE_SUB_THREADS 512
#define STBPE_SUB_MAX_BITS 8
// CHUNK: 8192 words, 16 registers of them per thread and three CTAs per SM; 16 384 where the table has so many ranges
// that a piece of 8192 words would leave less than one full load per range (more than six bits; 2^31 ids: 17.7 instead of
// 20.4 ms for this and the next pass, but 1.86 instead of 1.56 ms on 200 M ids).
template <int CHUNK>
__global__ void __launch_bounds__(STBPE_SUB_THREADS, CHUNK > 8192 ? 2 : 3) sub_partition_kernel(PartBuffers pb, int chunks_per_region, int sub_bits, uint16_t *__restrict__ offs) {
    extern __shared__ __align__(16) uint32_t s_out[];  // CHUNK words
    __shared__ unsigned int s_cnt[1 << STBPE_SUB_MAX_BITS], s_base[(1 << STBPE_SUB_MAX_BITS) + 1];
    constexpr int PER = CHUNK / STBPE_SUB_THREADS;
    const int D = 1 << sub_bits, lane = threadIdx.x & 31;
    // All regions' first pieces, then all second ones: the later pieces of a region, which has room for every token of its
    // share, are mostly empty, and would otherwise fall to the same CTAs (1.7 x 10^9 ids, four pieces: 23.5 ms, now 21.3).
    const i64 n_regions = (i64)STBPE_PARTS * pb.n_cta;
    for (i64 j = blockIdx.x; j < n_regions * chunks_per_region; j += gridDim.x) {
        const i64 piece = j / n_regions, region = j - piece * n_regions, chunk = region * chunks_per_region + piece, first = piece * CHUNK;
        const i64 left = (i64)pb.fill[region] - first;
        const int n = left <= 0 ? 0 : (left < CHUNK ? (int)left : CHUNK);
        uint32_t *w = pb.words + region * pb.cap + first;
        for (int i = threadIdx.x; i < D; i += STBPE_SUB_THREADS) s_cnt[i] = 0u;
        __syncthreads();
        uint32_t x[PER];
        uint16_t r[PER];
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int i = k * STBPE_SUB_THREADS + threadIdx.x;
            x[k] = i < n ? __ldcs(w + i) : 0u;
        }
#pragma unroll
        for (int k = 0; k < PER; ++k)
            if (k * STBPE_SUB_THREADS + (int)threadIdx.x < n)
                r[k] = (uint16_t)atomicAdd(&s_cnt[(x[k] << STBPE_PART_BITS) >> (32 - sub_bits)], 1u);
        __syncthreads();
        if (threadIdx.x < 32) {  // exclusive sums of the digits, D / 32 per lane (D >= 2)
            const int per = (D + 31) / 32;
            unsigned int own = 0;
            for (int k = 0; k < per; ++k) own += lane * per + k < D ? s_cnt[lane * per + k] : 0u;
            unsigned int incl = own;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const unsigned int o = __shfl_up_sync(0xFFFFFFFFu, incl, d);
                if (lane >= d) incl += o;
            }
            unsigned int at = incl - own;
            for (int k = 0; k < per; ++k)
                if (lane * per + k < D) {
                    s_base[lane * per + k] = at;
                    at += s_cnt[lane * per + k];
                }
            if (lane == 31) s_base[D] = incl;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < PER; ++k)
            if (k * STBPE_SUB_THREADS + (int)threadIdx.x < n) s_out[s_base[(x[k] << STBPE_PART_BITS) >> (32 - sub_bits)] + r[k]] = x[k];
        for (int i = threadIdx.x; i <= D; i += STBPE_SUB_THREADS) offs[chunk * (D + 1) + i] = (uint16_t)s_base[i];
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += STBPE_SUB_THREADS) w[i] = s_out[i];
        __syncthreads();
    }
}

// pass 3, one rank: the pair table, range by range.  A task is the range of words with one value of the first
// 8 + sub_bits bits; it owns `1 << task_bits` consecutive slots, which it fills in shared memory (word and
// 32-bit count) and writes out as they are, occupied or not: every slot of the table is written once with full
// lines, nothing is cleared before and no atomic reaches L2.  A word whose probe runs over the end of the range
// goes to the spill list, which is added to the finished table.
#define STBPE_BUILD_THREADS 512
__global__ void __launch_bounds__(STBPE_BUILD_THREADS, 3) build_table_kernel(EngineDev e, PartBuffers pb, int chunk_words, int chunks_per_region, int sub_bits, int task_bits,
                                                                          const uint16_t *__restrict__ offs, uint32_t *spill, unsigned int *n_spill,
                                                                          unsigned int spill_cap) {
    extern __shared__ __align__(16) uint32_t s_word[];
    const unsigned int TS = 1u << task_bits;
    unsigned int *s_num = s_word + TS;
    const int D = 1 << sub_bits, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n_tasks = STBPE_PARTS << sub_bits;
    const int shift = 32 - STBPE_PART_BITS - sub_bits - task_bits;
    for (int task = blockIdx.x; task < n_tasks; task += gridDim.x) {
        const uint32_t none = (uint32_t)(task ^ 1) << (32 - STBPE_PART_BITS - sub_bits);  // a word of another task
        for (unsigned int i = threadIdx.x; i < TS; i += STBPE_BUILD_THREADS) s_word[i] = none, s_num[i] = 0u;
        __syncthreads();
        const int p = task >> sub_bits, d = task & (D - 1);
        const int chunks = pb.n_cta * chunks_per_region;
        // A warp takes every sixteenth chunk, again first pieces before second ones (29.9 -> 23.5 ms on 1.7 x 10^9 ids).  Where a chunk's words are, each lane reads for another chunk, and the
        // next chunk's first words are on their way while one is counted: on 2^31 ids a chunk holds 32 words of
        // a range, and one dependent load after the other took 30 ms.
        constexpr int WARPS = STBPE_BUILD_THREADS / 32;
        for (int c0 = warp; c0 < chunks; c0 += 32 * WARPS) {
            const int c_own = c0 + lane * WARPS, n = min((chunks - c0 + WARPS - 1) / WARPS, 32);
            unsigned int own_lo = 0, own_hi = 0;
            i64 own_at = 0;
            if (c_own < chunks) {
                const i64 piece = c_own / pb.n_cta, region = (i64)p * pb.n_cta + c_own - piece * pb.n_cta, chunk = region * chunks_per_region + piece;
                own_lo = offs[chunk * (D + 1) + d], own_hi = offs[chunk * (D + 1) + d + 1];
                own_at = region * pb.cap + piece * chunk_words;
            }
            unsigned int next_lo = __shfl_sync(0xFFFFFFFFu, own_lo, 0), next_hi = __shfl_sync(0xFFFFFFFFu, own_hi, 0);
            const uint32_t *next_w = pb.words + __shfl_sync(0xFFFFFFFFu, own_at, 0);
            uint32_t first = next_lo + lane < next_hi ? __ldcs(next_w + next_lo + lane) : 0u;
            for (int j = 0; j < n; ++j) {
                const unsigned int lo = next_lo, hi = next_hi;
                const uint32_t *w = next_w;
                const uint32_t first_now = first;
                const int nj = j + 1 < n ? j + 1 : j;
                next_lo = __shfl_sync(0xFFFFFFFFu, own_lo, nj), next_hi = __shfl_sync(0xFFFFFFFFu, own_hi, nj);
                next_w = pb.words + __shfl_sync(0xFFFFFFFFu, own_at, nj);
                first = j + 1 < n && next_lo + lane < next_hi ? __ldcs(next_w + next_lo + lane) : 0u;
                // Four words per lane at a time, and a lane that has placed one goes on with its next at once: waiting for the
                // lane with the longest probe after every word took 5.5 turns a word, now 2.4 (200 M ids 1.06 ms, now 0.74).
                for (unsigned int i = lo; i < hi; i += 128) {
                    uint32_t q[4];
                    q[0] = i == lo ? first_now : i + lane < hi ? __ldcs(w + i + lane) : 0u;
#pragma unroll
                    for (int k = 1; k < 4; ++k) q[k] = i + k * 32 + lane < hi ? __ldcs(w + i + k * 32 + lane) : 0u;
                    int left = i + lane < hi ? min((int)(hi - i - lane + 31) / 32, 4) : 0;
                    unsigned int h = (q[0] >> shift) & (TS - 1);
                    while (__any_sync(0xFFFFFFFFu, left > 0)) {
                        if (left > 0) {
                            uint32_t k = ((volatile uint32_t *)s_word)[h];
                            if (k == none) {
                                k = atomicCAS(&s_word[h], none, q[0]);
                                if (k == none) k = q[0];
                            }
                            bool placed = k == q[0];
                            if (placed) {
                                atomicAdd(&s_num[h], 1u);
                            } else if (++h == TS) {
                                const unsigned int at = atomicAdd(n_spill, 1u);
                                if (at < spill_cap)
                                    spill[at] = q[0];
                                else
                                    atomicOr(&e.st->error, STBPE_DERR_DENSE_OVERFLOW);
                                placed = true;
                            }
                            if (placed) {
                                q[0] = q[1], q[1] = q[2], q[2] = q[3];
                                --left;
                                h = (q[0] >> shift) & (TS - 1);
                            }
                        }
                    }
                }
            }
        }
        __syncthreads();
        Slot *out = e.table + ((u64)task << task_bits);
        unsigned int keys = 0;
        for (unsigned int i = threadIdx.x; i < TS; i += STBPE_BUILD_THREADS) {
            Slot s;
            s.key = STBPE_EMPTY;
            s.count = (i64)s_num[i];
            if (s.count) {
                const uint32_t ab = unmix32(s_word[i]);
                s.key = ((u64)(ab >> 16) << 32) | (u64)(ab & 0xFFFFu);
                ++keys;
            }
            out[i] = s;
        }
        keys = __reduce_add_sync(0xFFFFFFFFu, keys);
        if (lane == 0 && keys) atomicAdd(&e.st->n_keys, (u64)keys);
        __syncthreads();
    }
}

__global__ void spill_to_table_kernel(EngineDev e, const uint32_t *__restrict__ spill, const unsigned int *n_spill, unsigned int spill_cap) {
    const unsigned int n = min(*n_spill, spill_cap);
    unsigned int fresh = 0;
    for (unsigned int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) part_word_to_table(e, spill[i], 1ull, fresh);
    if (fresh) atomicAdd(&e.st->n_keys, (u64)fresh);
}

// pass 2, several ranks, or one with a large table: partition p, owned by this rank, out of the regions of every rank.
// The grid of a partition is one wave of blocks whatever the number of ranks; a block walks over its share of the
// (source rank, region, half) units with one cache, which it adds to the table at the end.
__global__ void __launch_bounds__(1024)
    partition_table_peers_kernel(EngineDev e, WidePeers wp, int p_first, int p_step, int n_cta) {
    // consecutive groups of 2 * n_cta blocks take the partitions p_first, p_first + p_step, ...
    const int blocks_per_part = 2 * n_cta;
    const int p = p_first + (int)(blockIdx.x / blocks_per_part) * p_step;
    const int block = (int)(blockIdx.x % blocks_per_part);
    __shared__ uint32_t s_word[STBPE_PART_CACHE];
    __shared__ unsigned int s_cnt[STBPE_PART_CACHE];
    for (int i = threadIdx.x; i < STBPE_PART_CACHE; i += blockDim.x) {
        s_word[i] = 0xFFFFFFFFu;
        s_cnt[i] = 0u;
    }
    __syncthreads();
    unsigned int fresh = 0;
    const int n_units = wp.world * n_cta * 2;
    for (int unit = block; unit < n_units; unit += blocks_per_part) {
        const int half = unit & 1, region = (unit >> 1) % n_cta, src = (unit >> 1) / n_cta;
        const unsigned char *blk = wp.block[src];
        const WideHeader hd = *reinterpret_cast<const WideHeader *>(blk);
        if (hd.n_cta != n_cta) {  // every rank runs the first pass with the same grid
            if (threadIdx.x == 0) atomicOr(&e.st->error, STBPE_DERR_DENSE_OVERFLOW);
            continue;
        }
        const i64 n = wide_fill(blk)[(i64)p * n_cta + region];
        const uint32_t *w = wide_words(blk, n_cta) + ((i64)p * n_cta + region) * hd.cap;
        // words come four at a time (16-byte loads; regions are 16-byte aligned): a peer's words
        // cross NVLink, and one word per load left the loop waiting for the link's latency
        const i64 n4 = n / 4;
        const uint4 *w4 = reinterpret_cast<const uint4 *>(w);
        for (i64 i = (i64)half * blockDim.x + threadIdx.x; i <= n4; i += 2 * (i64)blockDim.x) {
            uint32_t x[4];
            int m = 4;
            if (i < n4) {
                const uint4 q = __ldcs(w4 + i);
                x[0] = q.x, x[1] = q.y, x[2] = q.z, x[3] = q.w;
            } else {
                m = (int)(n - n4 * 4);
                for (int k = 0; k < 4; ++k) x[k] = k < m ? w[n4 * 4 + k] : 0u;
            }
            for (int k = 0; k < m; ++k) {
                const unsigned int c = (x[k] * 0x9E3779B1u) >> (32 - STBPE_PART_CACHE_BITS);
                uint32_t kk = s_word[c];
                if (kk == 0xFFFFFFFFu && x[k] != 0xFFFFFFFFu) {
                    const uint32_t old = atomicCAS(&s_word[c], 0xFFFFFFFFu, x[k]);
                    kk = old == 0xFFFFFFFFu ? x[k] : old;
                }
                if (kk == x[k] && x[k] != 0xFFFFFFFFu)
                    atomicAdd(&s_cnt[c], 1u);
                else
                    part_word_to_table(e, x[k], 1ull, fresh);
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < STBPE_PART_CACHE; i += blockDim.x) {
        const unsigned int c = s_cnt[i];
        if (c) part_word_to_table(e, s_word[i], (u64)c, fresh);
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) fresh += __shfl_down_sync(0xFFFFFFFFu, fresh, d);
    if ((threadIdx.x & 31) == 0 && fresh) atomicAdd(&e.st->n_keys, (u64)fresh);
}

// hot pairs (both ids below 256) owned by this rank: the sum of every rank's counter
__global__ void dense_peers_to_table_kernel(EngineDev e, WidePeers wp, int n_cta) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= 65536) return;
    const u64 key = ((u64)(k >> 8) << 32) | (u64)(k & 0xFF);
    if (owner_of(key, wp.world) != wp.rank) return;
    u64 c = 0;
    for (int r = 0; r < wp.world; ++r) c += __ldcg(wide_dense(wp.block[r], n_cta) + k);
    if (c) sink_add<false>(e, key, (i64)c);
}
