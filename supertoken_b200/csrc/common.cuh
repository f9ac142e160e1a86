// Shared device-side definitions of the BPE merge-loop engine (sm_100a).
//
// Data layout in HBM
//   token stream : tiles of STBPE_TILE tokens, 16 bits each while every id fits 15 bits and 32 bits
//                  otherwise (stream.cuh).  The top bit of a token marks the first token of a row; a
//                  pair (i, j) of consecutive live tokens is countable iff token j does not carry
//                  that bit (rows are the only pair-breaking boundary, gpu_tokenizer/utils.py:586).
//                  A merge drops a token by overwriting it with the hole value (all ones), so it
//                  stores only the 16-byte units it changes; holes are squeezed out when a quarter
//                  of the stream is holes (repack_copy_kernel).
//   tile records : two versioned 32-byte records per tile {ver, len, first three live
//                  tokens, last two live tokens}.  During merge number m a tile is rewritten in
//                  place by exactly one warp, while the warps of neighbouring tiles need its
//                  PRE-merge head and tail.  A writer therefore fills the record with the older
//                  version and stamps it m; readers use the record with the largest
//                  version below m, which nobody writes during merge m.
//   pair table   : open addressing, linear probing, 16-byte slots {key = (a<<32)|b,
//                  int64 count}.  Keys are never removed; a count may return to zero.
//   candidates   : (one rank) the slots of all pairs at or above a threshold in selection order, a few
//                  hundred of the millions.  An add that lifts a pair over the threshold appends its
//                  slot, so the best pair is the best of the list until the list has run dry; then a
//                  scan of the table sets a lower threshold (candidate kernels in kernels.cuh).
//   block maxima : (several ranks) best (count, smallest key) of every block of slots.  An add that may
//                  change the maximum of its block sets the block's bit in a bitmap, and only those
//                  blocks are recomputed; the arg-max reduces the block maxima.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#define STBPE_TILE 1024  // tokens per tile: one warp owns a whole tile, 32 consecutive tokens per lane
#define STBPE_NONE 0xFFFFFFFFu
#define STBPE_FLAG 0x80000000u
#define STBPE_IDMASK 0x7FFFFFFFu
#define STBPE_EMPTY 0xFFFFFFFFFFFFFFFFull
#define STBPE_PROWS 16384  // rows of the pair filter: pair keys are hashed onto them (three hashes)
#define STBPE_PPITCH (STBPE_PROWS + 32)  // words per group of 32 tiles: the rows and the wildcard word (row STBPE_PROWS)
#define STBPE_MAX_PROBE (1u << 20)
#define STBPE_AUTO_PROBE (1u << 12)  // where the table grows instead: the longest probe to be expected at 90 % load is 3 000 slots

// device error bits
#define STBPE_DERR_TABLE_FULL 1u
#define STBPE_DERR_OUTBOX_FULL 2u
#define STBPE_DERR_LTABLE_FULL 4u
#define STBPE_DERR_KEY_MISSING 8u
#define STBPE_DERR_BAD_ID 16u
#define STBPE_DERR_TIMEOUT 32u
#define STBPE_DERR_DENSE_OVERFLOW 64u
#define STBPE_DERR_NARROW 128u  // an id does not fit the 16-bit stream: the host widens it and packs again

typedef unsigned long long u64;
typedef long long i64;

struct __align__(16) Slot {
    u64 key;
    i64 count;
};

struct __align__(16) TileRec {
    int ver;  // merge number that wrote this record; 0 = written at load; <0 = never written
    int len;  // live tokens when the record was written; exact below 3, otherwise only known to be >= 3
    uint32_t head[3];
    uint32_t tail;   // last live token
    uint32_t tail2;  // second to last live token (STBPE_NONE when len < 2)
    uint32_t pad;
};
static_assert(sizeof(TileRec) == 32, "merge_tile writes records word by word");

struct DevState {
    int cur_a, cur_b, cur_new;
    int filter_valid;          // the pair filter describes the stream: merges maintain it and skip tiles by it;
                               // 0 = stale (every merge visits every tile and leaves the filter alone)
    i64 cur_count;
    int merges_done, target, base_vocab, stopped;
    int stop_reason;
    int run_exit;              // why the last loop_kernel launch returned (STBPE_EXIT_*)
    unsigned int error;
    unsigned int max_id;       // largest id packed
    unsigned int ticket;
    int pad0;
    u64 n_keys;
    i64 n_live;
    i64 n_matches;             // of the last host-given merges (a launch that takes any starts at zero)
    u64 peek_key;
    i64 peek_count;
    i64 peek_ties;
    unsigned int n_ltouched;   // entries of the rank-local delta table awaiting the drain
    unsigned int n_lkept;      // entries the last drain had to keep (outbox chunk full)
    i64 export_n;
    int n_work;                // tiles visited by the last merge; < 0 = every tile
    unsigned int n_fixups;     // matches whose dropped token sits in another tile than their head (statistics)
    int exchange_only;         // multi-GPU: deltas still in flight, the next round only exchanges
    int round_incomplete;      // multi-GPU: this rank saw a full chunk or kept entries this round
    int forced_done;           // host-given merges the last loop_kernel launch applied
    int draws_used;            // outputs of the tie-breaking generator it used
    unsigned int n_cand;       // entries of the candidate list (may exceed its capacity: then it is incomplete)
    i64 theta_count;           // the list holds every pair with a larger count, or with this count and
    u64 theta_key;             // a key below this one
    int cand_state;            // STBPE_CAND_*
    int peek_valid;            // peek_key / peek_count are the best pair of the table as it stands
    // range a too coarse threshold search has to be continued in (cand_decide_kernel)
    i64 refine_lo, refine_hi;
    u64 refine_klo, refine_khi;
    i64 refine_above;          // pairs above the range
    u64 tile_bytes_in;         // merges: bytes of tiles and records read ...
    u64 tile_bytes_out;        // ... and bytes stored (rewritten 16-byte units and records), since the load
};
#define STBPE_TIES_OFFSET 512   // tied keys of ties_kernel lie this far behind the state
#define STBPE_TIES_CAP 1024
static_assert(sizeof(DevState) <= STBPE_TIES_OFFSET, "the tied keys follow the state");
#define STBPE_EXIT_STOP 0      // a stop rule fired (DevState::stop_reason) or the given merges are done
#define STBPE_EXIT_REPACK 1    // a quarter of the stream is holes
#define STBPE_EXIT_FILTER 2    // the pair filter starts to pay: build it
#define STBPE_EXIT_WIDEN 3     // the next id does not fit 15 bits
#define STBPE_EXIT_REFILL 4    // the candidate list has run dry or over
#define STBPE_EXIT_GROW 5      // the pair table fills up
#define STBPE_CAND_NONE 0      // no candidate list (fresh count)
#define STBPE_CAND_READY 1
#define STBPE_CAND_REFINE 2    // the threshold search needs another pass
#define STBPE_CAND_CAP 4096    // capacity of the candidate list
#define STBPE_CAND_MOST 1024   // a new threshold admits at most this many pairs ...
#define STBPE_CAND_LEAST 256   // ... and, if it can, at least this many
#define STBPE_CAND_BUCKETS 2048

// Synchronisation block of loop_kernel (loop.cuh), zeroed before every launch.
struct __align__(128) LoopSync {
    unsigned int arrived;                   // CTAs whose deltas are in the table, over all merges
    unsigned int pad0[31];
    unsigned int chosen;                    // CTAs that have read the candidates' counts, over all merges
    unsigned int pad1[31];
};

// Peer mailboxes (multi-GPU exchange over NVLink peer memory, no library collective).  Every rank owns
// one mailbox in its own HBM that its peers map: a header of flags and candidates followed by one
// inbox chunk per sender.  Flags carry the round number and only grow, so nothing is ever reset.
#define STBPE_MAX_PEERS 16
#define STBPE_MAIL_HEADER_BYTES 2048
struct MailHeader {
    u64 inbox_flag[STBPE_MAX_PEERS];     // [src] = last round whose chunk from src is complete here
    u64 cand_flag[STBPE_MAX_PEERS];      // [src] = last round whose candidate from src is here
    i64 cands[STBPE_MAX_PEERS][4];       // [src] = {key, count, incomplete, -}
    u64 round;                           // rounds this rank has committed (own use only)
    unsigned int out_count[STBPE_MAX_PEERS];  // entries sent to each owner this round (own use only)
};
static_assert(sizeof(MailHeader) <= STBPE_MAIL_HEADER_BYTES, "mailbox header does not fit");

struct EngineDev {
    unsigned char *mail[STBPE_MAX_PEERS];  // mailbox of every rank ([rank] = own), or null
    void *tiles;            // token stream: uint16_t or uint32_t tokens (stream.cuh)
    TileRec *recs;          // 2 per tile
    unsigned int *tile_live;  // live tokens per tile
    int n_tiles;
    Slot *table;
    u64 mask;
    unsigned int max_probe;  // slots an add looks at before it calls the table full
    int slot_bits;  // slot index bits below the table slice of a partition (slots = slices << slot_bits)
    unsigned int *cand;        // slots of the candidates
    unsigned int *cand_hist;   // STBPE_CAND_BUCKETS counters of the threshold search
    Slot *blockmax;
    unsigned int *dirty_bits;  // one bit per block
    unsigned int n_blocks;
    int blk_shift;             // log2 of the slots per block
    // presence[w * PPITCH + r]: bit t says "a pair whose key hashes to row r may have a token in tile
    // 32*w + t" (set when such a pair comes into being, never cleared until the next re-pack).  The rows
    // of 32 tiles lie together (64 KB): entering a pair stays inside one page, where a row-major layout
    // took a TLB miss per entry, and the look-up of a merge reads three words per 32 tiles.
    // A pair whose two tokens sit in different tiles is entered for both, so a merge finds every tile
    // it has to change by itself.  A Bloom filter with three hashes per pair: false positives
    // cost a wasted visit, never a missed one.  Row STBPE_PROWS is a wildcard: tiles that every
    // merge visits because the pair that starts at their last token is not known exactly (their
    // last token is the result of a run of equal tokens that ran on into the next tile).
    unsigned int *presence;
    DevState *st;
    LoopSync *sync;
    int32_t *merges;
    i64 *merge_counts;
    i64 *live_before;
    // multi-GPU: rank-local delta table, emptied into the per-owner outbox
    int world, rank;
    Slot *ltable;
    u64 lmask;
    unsigned int *ltouched;  // 2 lists of lslots entries: [0] filled by inserts, [1] by the drain
    Slot *outbox;  // [world][1 + cap] entries; entry 0 of a chunk = {count, 0}
    Slot *inbox;
    i64 cap_per_peer;
};

__device__ __forceinline__ MailHeader *mail_header(const EngineDev &e, int r) {
    return reinterpret_cast<MailHeader *>(e.mail[r]);
}
// chunk that rank `src` fills in the mailbox of rank `dst`
__device__ __forceinline__ Slot *mail_chunk(const EngineDev &e, int dst, int src) {
    return reinterpret_cast<Slot *>(e.mail[dst] + STBPE_MAIL_HEADER_BYTES) + (i64)src * (e.cap_per_peer + 1);
}

__device__ __forceinline__ u64 mix64(u64 x) {
    x ^= x >> 33;
    x *= 0xff51afd7ed558ccdULL;
    x ^= x >> 33;
    x *= 0xc4ceb9fe1a85ec53ULL;
    x ^= x >> 33;
    return x;
}


// Partition of a pair key: the top STBPE_PART_BITS bits of an invertible 32-bit mix of the key folded
// to 32 bits (for ids below 65 536 the fold is (a << 16) | b itself, so the mixed word identifies the
// pair).  One function places a key three ways: the partition is the top bits of its slot in the
// pair table (so the keys of a partition fill one contiguous slice of the table, which the
// partitioned first count keeps in L2 while it fills it), it is the partition of that count, and
// its residue modulo the number of ranks is the rank that owns the key.
#define STBPE_PART_BITS 8
#define STBPE_PARTS (1 << STBPE_PART_BITS)
__host__ __device__ __forceinline__ uint32_t mix32(uint32_t x) {
    x ^= x >> 16;
    x *= 0x7feb352du;
    x ^= x >> 15;
    x *= 0x846ca68bu;
    x ^= x >> 16;
    return x;
}
__host__ __device__ __forceinline__ uint32_t unmix32(uint32_t x) {  // inverse of mix32
    x ^= x >> 16;
    x *= 0x43021123u;
    x ^= (x >> 15) ^ (x >> 30);
    x *= 0x1d69e2a5u;
    x ^= x >> 16;
    return x;
}
__host__ __device__ __forceinline__ uint32_t fold_key(u64 key) {
    const uint32_t a = (uint32_t)(key >> 32), b = (uint32_t)key;
    return (a << 16) ^ b ^ ((a >> 16) * 0x9E3779B1u) ^ ((b >> 16) * 0x85EBCA77u);
}
__host__ __device__ __forceinline__ unsigned int part_of(u64 key) {
    return mix32(fold_key(key)) >> (32 - STBPE_PART_BITS);
}

__device__ __forceinline__ int owner_of(u64 key, int world) {
    return (int)(part_of(key) % (unsigned int)world);
}

// Table slice of a partition.  A rank holds only the keys it owns, i.e. the partitions with its
// residue modulo the number of ranks: their slices are numbered densely (partition / ranks), so the
// whole table is in use whatever the number of ranks.
__device__ __forceinline__ unsigned int slice_of(const EngineDev &e, unsigned int part) {
    return e.world == 1 ? part : part / (unsigned int)e.world;
}
__device__ __forceinline__ unsigned int hash32(u64 key) {
    unsigned int a = (unsigned int)(key >> 32), b = (unsigned int)key;
    unsigned int h = a * 0x9E3779B1u ^ (b * 0x85EBCA77u + 0x7F4A7C15u);
    h ^= h >> 15;
    h *= 0x2C1B3C6Du;
    h ^= h >> 13;
    return h;
}

// First slot probed for a key: its partition's slice, then the bits of the mix below the partition's.  With one
// rank that is the mixed word shifted right, so the slots of a range of words are contiguous (wide_count.cuh
// builds the table range by range).
__device__ __forceinline__ u64 slot_of_word(const EngineDev &e, uint32_t word) {
    const u64 top = (u64)slice_of(e, word >> (32 - STBPE_PART_BITS)) << e.slot_bits;
    return top | (u64)((word << STBPE_PART_BITS) >> (32 - e.slot_bits));
}
__device__ __forceinline__ u64 slot_of(const EngineDev &e, u64 key) { return slot_of_word(e, mix32(fold_key(key))); }

__device__ __forceinline__ bool better(u64 k1, i64 c1, u64 k2, i64 c2) {
    // (k1, c1) beats (k2, c2): larger count, ties to the smaller packed key
    // (gpu_tokenizer/trainers/bpe_gpu.py:106-127)
    return c1 > c2 || (c1 == c2 && k1 < k2);
}

// The host and every kernel read mutable state through L2: loop_kernel keeps running while other
// SMs write it, and the L1 caches are not coherent.
__device__ __forceinline__ Slot ldcg_slot(const Slot *p) {
    const uint4 raw = __ldcg(reinterpret_cast<const uint4 *>(p));
    Slot s;
    s.key = ((u64)raw.y << 32) | raw.x;
    s.count = (i64)(((u64)raw.w << 32) | raw.z);
    return s;
}

__device__ __forceinline__ void mark_dirty(const EngineDev &e, u64 slot_index) {
    const unsigned int blk = (unsigned int)(slot_index >> e.blk_shift);
    atomicOr(&e.dirty_bits[blk >> 5], 1u << (blk & 31));  // result unused: a reduction
}

// threshold of the candidate list in selection order: a larger count, or the same count and a key below `key`
struct Theta {
    i64 count;
    u64 key;
    __device__ __forceinline__ bool admits(i64 c, u64 k) const { return c > count || (c == count && k < key); }
};

// Whether a probe of the pair table goes on: a long one stops when another has found the table full.  (Otherwise every
// add to a full table walks `max_probe` slots: 2.5e8 ids into 2^25 slots took 2.5 minutes to report it.)
__device__ __forceinline__ bool probe_on(const EngineDev &e, unsigned int probe) {
    return probe < e.max_probe && ((probe & 255u) != 255u || !(*(volatile unsigned int *)&e.st->error & STBPE_DERR_TABLE_FULL));
}

// Add delta to key in the pair table, inserting the key when absent.  `fresh` counts inserted keys
// (the caller adds them to DevState::n_keys).  `made`: the key probably does not exist yet, so the first
// access is the compare-and-swap that claims a slot instead of a load that would find it empty.
// NOTE says what the arg-max has to learn of the add:
//   NOTE_NONE   nothing (first counts: candidates / maxima are built afterwards)
//   NOTE_CAND   the add that lifts a pair over the candidates' threshold appends its slot to the list.  Only
//               adds look at the count they leave; a subtraction never lifts a pair.
//   NOTE_DIRTY  the maximum of the slot's block can only change if this key is the recorded maximum or if its
//               count now reaches it (the recorded maxima do not change while deltas are applied).  An add sees
//               a count that is at least the key's final one when subtractions of the same key follow
//               it, so the check after adds alone is enough.
enum { NOTE_NONE, NOTE_CAND, NOTE_DIRTY };
template <int NOTE>
__device__ __forceinline__ void table_add(const EngineDev &e, u64 key, i64 delta, bool made, unsigned int &fresh,
                                          const Theta &theta = Theta()) {
    u64 h = slot_of(e, key);
    const u64 blk = h >> e.blk_shift;
    Slot mx;
    if (NOTE == NOTE_DIRTY) mx = ldcg_slot(e.blockmax + blk);  // fetched together with the first probe
#pragma unroll 1
    for (unsigned int probe = 0; probe_on(e, probe); ++probe) {
        Slot *s = &e.table[h];
        u64 k = made ? STBPE_EMPTY : __ldcg(&s->key);
        if (k == STBPE_EMPTY) {
            k = atomicCAS(&s->key, STBPE_EMPTY, key);
            if (k == STBPE_EMPTY) {
                ++fresh;
                k = key;
            }
        }
        if (k == key) {
            if (NOTE == NOTE_NONE || (NOTE == NOTE_CAND && delta < 0)) {
                atomicAdd((u64 *)&s->count, (u64)delta);  // result unused: a reduction
                return;
            }
            const i64 was = (i64)atomicAdd((u64 *)&s->count, (u64)delta), now = was + delta;
            if (NOTE == NOTE_CAND) {
                if (theta.admits(now, key) && !theta.admits(was, key)) {
                    const unsigned int i = atomicAdd(&e.st->n_cand, 1u);
                    if (i < STBPE_CAND_CAP) e.cand[i] = (unsigned int)h;
                }
            } else {
                if ((h >> e.blk_shift) != blk) mx = ldcg_slot(e.blockmax + (h >> e.blk_shift));
                if (key == mx.key || (delta > 0 && (now > mx.count || (now == mx.count && key < mx.key)))) mark_dirty(e, h);
            }
            return;
        }
        h = (h + 1) & e.mask;
    }
    atomicOr(&e.st->error, STBPE_DERR_TABLE_FULL);
}

// rank-local delta table (multi-GPU): same probing, first touch recorded for the drain
__device__ __forceinline__ void ltable_add(const EngineDev &e, u64 key, i64 delta) {
    u64 h = mix64(key * 0x9E3779B97F4A7C15ULL + 1) & e.lmask;
#pragma unroll 1
    for (unsigned int probe = 0; probe <= (unsigned int)e.lmask; ++probe) {
        Slot *s = &e.ltable[h];
        u64 k = *(volatile u64 *)&s->key;
        if (k == STBPE_EMPTY) {
            u64 old = atomicCAS(&s->key, STBPE_EMPTY, key);
            if (old == STBPE_EMPTY) {
                unsigned int i = atomicAdd(&e.st->n_ltouched, 1u);
                e.ltouched[i] = (unsigned int)h;  // i <= lmask: one entry per slot
                k = key;
            } else {
                k = old;
            }
        }
        if (k == key) {
            atomicAdd((u64 *)&s->count, (u64)delta);
            return;
        }
        h = (h + 1) & e.lmask;
    }
    atomicOr(&e.st->error, STBPE_DERR_LTABLE_FULL);
}

// first counts: into the rank-local delta table, or straight into the pair table
template <bool MG>
__device__ __forceinline__ void sink_add(const EngineDev &e, u64 key, i64 delta) {
    if (MG) {
        ltable_add(e, key, delta);
    } else {
        unsigned int fresh = 0;
        table_add<NOTE_NONE>(e, key, delta, false, fresh);
        if (fresh) atomicAdd(&e.st->n_keys, (u64)fresh);
    }
}

// ---------------------------------------------------------------------------------------
// Per-CTA aggregation table in shared memory: key -> int32 delta.  Inserts that do not
// find a slot within a few probes go straight to the global sink.
// The table is addressed through the shared state space explicitly (ld/atom/red .shared):
// atomics issued through generic pointers to shared memory were measured at ~450 cycles each
// on this part, against ~10-20 for the .shared forms.
// ---------------------------------------------------------------------------------------
struct SmemTable {
    u64 *keys;
    int *vals;
    unsigned int mask;
};

__device__ __forceinline__ u64 lds_u64_volatile(const u64 *p) {
    u64 v;
    asm volatile("ld.volatile.shared.u64 %0, [%1];" : "=l"(v) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
    return v;
}
__device__ __forceinline__ u64 atoms_cas_u64(u64 *p, u64 cmp, u64 val) {
    u64 old;
    asm volatile("atom.shared.cas.b64 %0, [%1], %2, %3;"
                 : "=l"(old)
                 : "r"((uint32_t)__cvta_generic_to_shared(p)), "l"(cmp), "l"(val)
                 : "memory");
    return old;
}
__device__ __forceinline__ void reds_add_s32(int *p, int v) {
    asm volatile("red.shared.add.s32 [%0], %1;" ::"r"((uint32_t)__cvta_generic_to_shared(p)), "r"(v) : "memory");
}

__device__ __forceinline__ void smem_table_clear(const SmemTable &t) {
    for (unsigned int i = threadIdx.x; i <= t.mask; i += blockDim.x) {
        t.keys[i] = STBPE_EMPTY;
        t.vals[i] = 0;
    }
}

// pair filter: the three rows of a pair key, and setting the pair's bits for a tile.  The filter is
// kept only while it pays: a merge with more matches than tiles visits nearly every tile anyway, and
// entering its new pairs costs more than the whole rewrite (measured: 37 of 61 ms on the first 20
// merges of a 1 GiB corpus), so the host lets the filter go stale for such merges and rebuilds it
// from the stream once the counts have fallen below the number of tiles.  With about a
// thousand distinct pairs in a full tile, three bits per pair over 16 384 rows leave a row about 17 %
// full and let through about 0.5 % of the tiles that do not hold the pair (two bits over 8 192 rows
// let through 5 %, which late in a run was most of the tiles a merge visited).
__device__ __forceinline__ void filter_rows(u64 key, unsigned int &r1, unsigned int &r2, unsigned int &r3) {
    // 32-bit arithmetic only (a 64-bit finaliser costs about three times the instructions, and the
    // merge kernel hashes two keys per match): two rows from disjoint bits of one mixed word, the
    // third from a second multiplicative mix of it
    const unsigned int h = hash32(key);
    unsigned int g = h * 0x9E3779B1u;
    g ^= g >> 15;
    r1 = h & (STBPE_PROWS - 1);
    r2 = (h >> 14) & (STBPE_PROWS - 1);
    r3 = (g >> 9) & (STBPE_PROWS - 1);
}
// enter a pair for the tiles of its two tokens (tile2 < 0: one tile)
__device__ __forceinline__ void filter_set(const EngineDev &e, int tile, int tile2, u64 key) {
    unsigned int r1, r2, r3;
    filter_rows(key, r1, r2, r3);
#pragma unroll 1
    for (;;) {
        unsigned int *g = e.presence + (size_t)((unsigned int)tile >> 5) * STBPE_PPITCH;
        const unsigned int bit = 1u << (tile & 31);
        // results unused: reductions, nothing waits for them
        atomicOr(g + r1, bit);
        atomicOr(g + r2, bit);
        atomicOr(g + r3, bit);
        if (tile2 < 0 || tile2 == tile) return;
        tile = tile2;
    }
}

// slow path: probe for the key, claim an empty slot, or give up after a few probes
template <bool MG>
__device__ __noinline__ void smem_table_add_probe(SmemTable t, const EngineDev *e, u64 key, int delta,
                                                  unsigned int h) {
#pragma unroll 1
    for (int probe = 0; probe < 8; ++probe) {
        u64 k = lds_u64_volatile(&t.keys[h]);
        if (k == STBPE_EMPTY) {
            const u64 old = atoms_cas_u64(&t.keys[h], STBPE_EMPTY, key);
            k = (old == STBPE_EMPTY) ? key : old;
        }
        if (k == key) {
            reds_add_s32(&t.vals[h], delta);
            return;
        }
        h = (h + 1) & t.mask;
    }
    sink_add<MG>(*e, key, (i64)delta);
}

// A key never leaves its slot once written, so a plain load that sees the key is final; any
// other value (empty or a different key) goes to the probing path.  Keeping the fast path free
// of volatile accesses lets several independent adds overlap.
__device__ __forceinline__ u64 lds_u64(const u64 *p) {
    u64 v;
    asm("ld.shared.u64 %0, [%1];" : "=l"(v) : "r"((uint32_t)__cvta_generic_to_shared(p)));
    return v;
}
template <bool MG>
__device__ __forceinline__ void smem_table_add(const SmemTable &t, const EngineDev &e, u64 key,
                                               int delta) {
    const unsigned int h = hash32(key) & t.mask;
    if (lds_u64(&t.keys[h]) == key)
        reds_add_s32(&t.vals[h], delta);
    else
        smem_table_add_probe<MG>(t, &e, key, delta, h);
}

template <bool MG>
__device__ __forceinline__ void smem_table_flush(const SmemTable &t, const EngineDev &e) {
    for (unsigned int i = threadIdx.x; i <= t.mask; i += blockDim.x) {
        u64 k = t.keys[i];
        int v = t.vals[i];
        if (k != STBPE_EMPTY && v != 0) sink_add<MG>(e, k, (i64)v);
    }
}

// ---------------------------------------------------------------------------------------
// Tile records
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ TileRec load_rec(const TileRec *p) {
    TileRec r;
    const uint4 *q = reinterpret_cast<const uint4 *>(p);
    const uint4 x = __ldcg(q), y = __ldcg(q + 1);
    r.ver = (int)x.x;
    r.len = (int)x.y;
    r.head[0] = x.z;
    r.head[1] = x.w;
    r.head[2] = y.x;
    r.tail = y.y;
    r.tail2 = y.z;
    r.pad = 0;
    return r;
}

// record of `tile` that was current before merge number m; returns its slot index
__device__ __forceinline__ int current_rec(const EngineDev &e, int tile, int m, TileRec &out) {
    TileRec r0 = load_rec(&e.recs[2 * tile]);
    TileRec r1 = load_rec(&e.recs[2 * tile + 1]);
    bool ok0 = r0.ver >= 0 && r0.ver < m;
    bool ok1 = r1.ver >= 0 && r1.ver < m;
    int s = (ok1 && (!ok0 || r1.ver > r0.ver)) ? 1 : 0;
    out = s ? r1 : r0;
    if (!ok0 && !ok1) out.len = 0;
    return s;
}

// Live tokens around a tile, in stream order: the last two live tokens before it and the next three
// after it (STBPE_NONE where the stream ends), with the tiles that hold prev, nxt[0] and nxt[1].
struct Halo {
    uint32_t prev, prev2, nxt[3];
    int prev_tile, next_tile, next2_tile;
};

// Walks records only; for tiles whose neighbours hold too few tokens to answer by themselves.
static __device__ __noinline__ void gather_halo(const EngineDev &e, int tile, int m, Halo &h) {
    h.prev_tile = h.next_tile = h.next2_tile = -1;
    h.prev = h.prev2 = STBPE_NONE;
    h.nxt[0] = h.nxt[1] = h.nxt[2] = STBPE_NONE;
    TileRec r;
    int back = 0;
    for (int t = tile - 1; t >= 0 && back < 2; --t) {
        current_rec(e, t, m, r);
        if (r.len > 0) {
            if (back == 0) {
                h.prev = r.tail;
                h.prev_tile = t;
                back = 1;
                if (r.len > 1) {
                    h.prev2 = r.tail2;
                    back = 2;
                }
            } else {
                h.prev2 = r.tail;
                back = 2;
            }
        }
    }
    int have = 0;
    for (int t = tile + 1; t < e.n_tiles && have < 3; ++t) {
        current_rec(e, t, m, r);
        const int take = r.len < 3 ? r.len : 3;
        for (int i = 0; i < take && have < 3; ++i) {
            if (have == 0) h.next_tile = t;
            if (have == 1) h.next2_tile = t;
            h.nxt[have++] = r.head[i];
        }
    }
}

// first live token after a tile, from the records (general count, filter build)
__device__ __forceinline__ uint32_t first_after(const EngineDev &e, int tile, int m) {
    for (int t = tile + 1; t < e.n_tiles; ++t) {
        TileRec r;
        current_rec(e, t, m, r);
        if (r.len > 0) return r.head[0];
    }
    return STBPE_NONE;
}
// last live token before a tile
__device__ __forceinline__ uint32_t last_before(const EngineDev &e, int tile, int m) {
    for (int t = tile - 1; t >= 0; --t) {
        TileRec r;
        current_rec(e, t, m, r);
        if (r.len > 0) return r.tail;
    }
    return STBPE_NONE;
}
