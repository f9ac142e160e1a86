// Host side of the C ABI declared in include/stbpe.h: memory, launches, maintenance between them.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <cuda_runtime.h>
#include <dlfcn.h>
#include <nccl.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/stbpe.h"
#include "host_copy.h"
#include "kernels.cuh"
#include "loop.cuh"

#include <algorithm>
#include <mutex>
#include <utility>

#define STBPE_PINNED_BYTES ((size_t)4 << 20)
#define STBPE_PINNED_STATE 16384  // bytes in front that the device state travels through
#define STBPE_COUNT_SMEM (STBPE_COUNT_SLOTS * 12)
#define STBPE_MAX_SLOTS (1ll << 32)  // of one rank's pair table

#define STBPE_VISIBLE __attribute__((visibility("default")))

struct stbpe_engine {
    stbpe_config cfg;
    EngineDev d;
    i64 max_tokens, n_tokens;
    int max_tiles;
    bool wide;            // the stream holds 32-bit tokens (an id does not fit 15 bits)
    size_t tiles_bytes, alt_bytes;  // sizes of the two stream buffers
    u64 slots;
    Slot *partial;
    i64 *cand;
    u64 lslots;
    int sm_count;
    int select_grid, refresh_grid;
    size_t count_smem;
    int2 *forced;         // device copy of host-given merges
    uint32_t *draws;      // STBPE_DRAWS outputs of a tie-breaking generator, from the first call that brings any
    int forced_cap;
    bool recs_stale, counted;
    bool filter_valid;    // host mirror of DevState::filter_valid
    double filter_density;  // the filter is kept while (matches of the last merge) <= filter_density x tiles
    u64 *dense;           // 65 536 global counters of the byte-level count path
    PartBuffers parts;    // partition buffers of the 16-bit-vocabulary count path (allocated at first use)
    unsigned char *wide_block;             // their allocation: header, fills, hot counters, regions
    u64 *wide_dense;                       // the hot counters inside it
    void *wide_mapped[STBPE_MAX_PEERS];    // peers' allocations as mapped into this process
    WidePeers wide_peers;
    bool wide_open, wide_counted;          // peers mapped / the table holds a count made by stbpe_mg_wide_pass2
    bool full_refresh_pending;             // that count marked no block dirty: the next refresh recomputes all maxima
    i64 dense32_min;      // streams shorter than this use the general kernel; < 0: by the rule of wide_eligible
    i64 narrow_counts;    // the merge loop on 16-bit tokens compares counts below this
    bool only_bytes;      // every token so far came from stbpe_append_bytes (ids < 256)
    ncclComm_t comm;      // own NCCL communicator for the native multi-GPU round loop
    i64 *all_cands;       // world x 4 gathered candidates (native loop)
    bool own_boxes;
    unsigned char *mail_own;               // this rank's mailbox (peer-memory rounds)
    void *mail_mapped[STBPE_MAX_PEERS];    // peers' mailboxes as mapped into this process
    bool peers_open;
    bool count_timed;     // ev0 / ev1 span the histogram kernels of the last count; not yet read into count_ms
    float count_ms;       // device time of the histogram kernels of the last count
    float convert_ms;     // device time of moving a dense histogram into the pair table (wide path)
    cudaEvent_t ev0, ev1;
    void *tiles_alt;  // second stream buffer of the re-pack (at creation when memory allows)
    i64 *rp_lens, *rp_offs;  // re-pack scratch: tile lengths and their exclusive sums
    void *rp_tmp;
    size_t rp_tmp_bytes;
    int repacks;
    int repacks_since_load;
    cudaGraphExec_t graph;  // a batch of peer-memory rounds (several ranks)
    int graph_tiles_n;
    void *graph_tiles, *graph_filter;
    bool graph_wide;
    bool use_graph;
    int part_group;       // partitions per launch of the second pass of the partitioned count
    std::string err;
    std::vector<stbpe::Block> allocs;
    bool broken;          // a CUDA call failed: work of this engine may still be pending
    stbpe::Block pinned;  // host side of small transfers: the device state, then small inputs
    bool sync_zeroed;     // the barrier counters of the next loop launch are zero: each launch clears the other pair
    int sync_turn;
    bool cand_stale;      // the candidate list is used up: collect one before the next choice
    bool foreign_ids;     // a merge of the caller's may have brought an id of 65 536 or more
    unsigned int max_id;  // largest id appended through stbpe_append_ids
    i64 bytes_below, made_below;  // the stream's bytes, and the ids that merges have brought, lie below these
    unsigned int load_err;  // error bits of the rows appended so far
    bool merges_known;    // merges_done mirrors the device (several host-driven merges in a row)
    int merges_done;
    bool state_stale;     // the device state is that of a stream that has been dropped
    bool table_auto;      // the table is sized by the stream and grows with the keys
    u64 table_cap;        // slots the allocated table has room for
    u64 slots_needed;     // a count of this stream has overflowed a quarter of these
    size_t presence_cap;  // groups of 32 tiles the pair filter has room for
    void *off_dev;        // row offsets of an append
    size_t off_cap;
};

// what differs between GPUs, asked once per device
struct DeviceInfo {
    int sm_count = 0;
    cudaError_t err = cudaSuccess;
    const char *what = "";
};
extern "C" {
static const DeviceInfo &device_info(int dev);
}

static thread_local std::string g_create_err;
namespace { struct NcclApi; NcclApi &nccl_api(); }

static int fail(stbpe_engine *e, int code, const std::string &msg) {
    if (e)
        e->err = msg;
    else
        g_create_err = msg;
    return code;
}

static int cuda_fail(stbpe_engine *e, cudaError_t c, const char *what) {
    std::string m = std::string(what) + ": " + cudaGetErrorString(c);
    if (c == cudaErrorMemoryAllocation) m = "CUDA out of memory (" + m + ")";
    cudaGetLastError();
    if (e) e->broken = true;
    return fail(e, STBPE_E_CUDA, m);
}

#define CK(call)                                                  \
    do {                                                          \
        cudaError_t c_ = (call);                                  \
        if (c_ != cudaSuccess) return cuda_fail(e, c_, #call);    \
    } while (0)

// Memory of an engine.  One-rank engines share the block cache; the buffers of several ranks are mapped by other
// processes (CUDA IPC) and stay plain allocations.
template <typename T>
static cudaError_t dev_alloc(stbpe_engine *e, T **p, size_t count) {
    stbpe::Block b;
    const size_t bytes = count * sizeof(T) > 0 ? count * sizeof(T) : 16;
    cudaError_t c = cudaSuccess;
    if (e->cfg.world_size > 1) {
        c = cudaMalloc(&b.p, bytes);
        b.size = bytes;
    } else {
        c = stbpe::device_blocks().get(e->cfg.device, bytes, &b);
    }
    if (c == cudaSuccess) {
        e->allocs.push_back(b);
        *p = reinterpret_cast<T *>(b.p);
    }
    return c;
}

static void give_back(stbpe_engine *e, const stbpe::Block &b) {
    if (e->cfg.world_size > 1 || e->broken)
        cudaFree(b.p);
    else
        stbpe::device_blocks().put(e->cfg.device, b);
}

// no work that uses the memory may be pending
static void dev_free(stbpe_engine *e, void *p) {
    if (!p) return;
    for (auto &q : e->allocs)
        if (q.p == p) {
            give_back(e, q);
            q = e->allocs.back();
            e->allocs.pop_back();
            return;
        }
}

// pieces of one allocation
struct Arena {
    std::vector<std::pair<void **, size_t>> parts;
    size_t total = 0;
    template <typename T>
    void add(T **p, size_t count) {
        parts.push_back({reinterpret_cast<void **>(p), total});
        total += (count * sizeof(T) + 255) & ~(size_t)255;
    }
    cudaError_t alloc(stbpe_engine *e) {
        unsigned char *base = nullptr;
        const cudaError_t c = dev_alloc(e, &base, total);
        if (c == cudaSuccess)
            for (auto &q : parts) *q.first = base + q.second;
        return c;
    }
};

static u64 next_pow2(u64 x) {
    u64 p = 1;
    while (p < x) p <<= 1;
    return p;
}

// Calls f(uint16_t{}) or f(uint32_t{}) for the engine's stream.
template <typename F>
static auto with_tok(const stbpe_engine *e, F &&f) {
    return e->wide ? f(uint32_t{}) : f(uint16_t{});
}
// Whether a fresh stream starts with 32-bit tokens.  Several ranks run rounds without a look from the host, so
// there the ids of all merges must fit from the start; a single rank widens its stream when it gets there.
static bool starts_wide(const stbpe_config &c) {
    const i64 last = (i64)c.base_vocab + (c.world_size > 1 ? c.max_merges : 0);
    return last >= (i64)Tok<uint16_t>::IDMASK;
}
static size_t tok_bytes(const stbpe_engine *e) { return e->wide ? 4 : 2; }

// Every id of the stream lies below this.
static i64 ids_below(const stbpe_engine *e) {
    return std::max({e->bytes_below, e->made_below, e->only_bytes ? (i64)0 : (i64)e->max_id + 1});
}

// log2 of the tiles a CTA takes together from the pair filter: eight once every CTA gets several units, fewer on
// smaller streams, so that the visited tiles spread over all CTAs.  (Whole words of the filter, 32 tiles, are fewer
// loads, but where the tiles that hold a pair lie together one CTA gets many of them: on the adversarial corpus the
// others waited 20-30 us of a step of 80.)
static int unit_shift(const stbpe_engine *e, int grid) {
    int sh = 3;
    while (sh > 0 && (((i64)e->d.n_tiles + (1 << sh) - 1) >> sh) < 2 * (i64)grid) --sh;
    return sh;
}

extern "C" {

STBPE_VISIBLE const char *stbpe_version(void) { return "stbpe 0.2 (sm_100a)"; }

STBPE_VISIBLE const char *stbpe_last_error(const stbpe_engine *e) {
    return e ? e->err.c_str() : g_create_err.c_str();
}

STBPE_VISIBLE int stbpe_destroy(stbpe_engine *e) {
    if (!e) return STBPE_OK;
    cudaSetDevice(e->cfg.device);
    if (e->graph) cudaGraphExecDestroy(e->graph);
    for (void *&m : e->mail_mapped)
        if (m) {
            cudaIpcCloseMemHandle(m);
            m = nullptr;
        }
    for (void *&m : e->wide_mapped)
        if (m) {
            cudaIpcCloseMemHandle(m);
            m = nullptr;
        }
    // the NCCL communicator is shared by the engines of this process and lives until exit
    if (e->ev0) cudaEventDestroy(e->ev0);
    if (e->ev1) cudaEventDestroy(e->ev1);
    // every entry point of a one-rank engine ends synchronised, so nothing is pending unless a call failed
    if (e->broken) cudaDeviceSynchronize();
    for (const stbpe::Block &b : e->allocs) give_back(e, b);
    stbpe::pinned_blocks().put(0, e->pinned);
    delete e;
    return STBPE_OK;
}

STBPE_VISIBLE int stbpe_trim(int32_t device, int64_t keep_bytes) {
    if (device < -1 || device >= 64 || keep_bytes < 0) return STBPE_E_BADARG;
    if (device < 0)
        stbpe::pinned_blocks().trim(0, (size_t)keep_bytes);
    else
        stbpe::device_blocks().trim(device, (size_t)keep_bytes);
    return STBPE_OK;
}

static const DeviceInfo &device_info(int dev) {
    static std::mutex mu;
    static DeviceInfo infos[64];
    static bool known[64] = {};
    const int k = dev >= 0 && dev < 64 ? dev : 0;
    std::lock_guard<std::mutex> lock(mu);
    DeviceInfo &i = infos[k];
    if (known[k] && i.err == cudaSuccess) return i;
    known[k] = true;
    int optin = 0;
    i.what = "cudaDeviceGetAttribute";
    i.err = cudaDeviceGetAttribute(&i.sm_count, cudaDevAttrMultiProcessorCount, dev);
    if (i.err == cudaSuccess) i.err = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (i.err != cudaSuccess) return i;
    // kernels that use more shared memory than the default limit
    i.what = "cudaFuncSetAttribute";
#define SMEM(kern, bytes) \
    if (i.err == cudaSuccess) i.err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(bytes))
    SMEM((merge_kernel<uint16_t, false>), MergeGeom<uint16_t>::BYTES);
    SMEM((merge_kernel<uint16_t, true>), MergeGeom<uint16_t>::BYTES);
    SMEM((merge_kernel<uint32_t, false>), MergeGeom<uint32_t>::BYTES);
    SMEM((merge_kernel<uint32_t, true>), MergeGeom<uint32_t>::BYTES);
    SMEM((loop_kernel<uint16_t, FILTER_OFF, 9>), optin - 4096);
    SMEM((loop_kernel<uint16_t, FILTER_OFF, 11>), optin - 4096);
    SMEM((loop_kernel<uint16_t, FILTER_OFF, 15>), optin - 4096);
    SMEM((loop_kernel<uint16_t, FILTER_ON, 11>), optin - 4096);
    SMEM((loop_kernel<uint16_t, FILTER_ON, 13>), optin - 4096);
    SMEM((loop_kernel<uint16_t, FILTER_ON, 15>), optin - 4096);
    SMEM((loop_kernel<uint16_t, FILTER_OFF, 15, true>), optin - 4096);
    SMEM((loop_kernel<uint16_t, FILTER_ON, 15, true>), optin - 4096);
    SMEM((loop_kernel<uint32_t, FILTER_OFF, 15>), optin - 4096);
    SMEM((loop_kernel<uint32_t, FILTER_ON, 15>), optin - 4096);
    SMEM((count_kernel<uint16_t, false>), STBPE_COUNT_SMEM);
    SMEM((count_kernel<uint16_t, true>), STBPE_COUNT_SMEM);
    SMEM((count_kernel<uint32_t, false>), STBPE_COUNT_SMEM);
    SMEM((count_kernel<uint32_t, true>), STBPE_COUNT_SMEM);
    SMEM(count_dense_kernel<uint16_t>, 32768 * 4);
    SMEM(count_dense_kernel<uint32_t>, 32768 * 4);
    SMEM(partition_pairs_kernel<uint16_t>, STBPE_PART_SMEM_BYTES);
    SMEM(partition_pairs_kernel<uint32_t>, STBPE_PART_SMEM_BYTES);
    SMEM(sub_partition_kernel<16384>, 16384 * sizeof(uint32_t));
    SMEM(build_table_kernel, 8 << 13);
    SMEM(presence_rebuild_kernel<uint16_t>, STBPE_PROWS * sizeof(unsigned int));
    SMEM(presence_rebuild_kernel<uint32_t>, STBPE_PROWS * sizeof(unsigned int));
#undef SMEM
    return i;
}

// Slots of a table that is sized by the stream.
// One rank: for the first count of n ids below `ids`; a count that does not fit takes four times as many (stbpe_count_initial), merges
// grow the table (grow_table).  Of Zipf ids over 65 536, 42 % of 2^20 pairs are distinct, 17 % of 2^27, 8 % of 2^31: a slot
// per token up to 2^25 of them, one for four tokens of long streams, up to 2^29 (8 GiB); no more than pairs can differ.
static u64 auto_slots(i64 n, i64 ids) {
    u64 slots = std::max((u64)std::min(n, (i64)1 << 25), (u64)n / 4);
    if (ids < 65536) slots = std::min(slots, 2 * (u64)ids * (u64)ids);
    return std::min(std::max(slots, (u64)1 << 20), (u64)1 << 29);
}
// Several ranks: keys are never removed and nothing grows, so it must hold every pair a run ever creates; 2^27 slots
// carried 32 000 merges on 2^30 tokens, streams of 2^32 tokens and more get 2^29 (8 GiB).
static u64 auto_slots_mg(i64 max_tokens) {
    const u64 cap = max_tokens >= (1ll << 32) ? (1ull << 29) : (1ull << 27);
    return std::min(std::max((u64)max_tokens / 4, (u64)1 << 20), cap);
}

static void set_slots(stbpe_engine *e, u64 want) {
    const u64 slots = next_pow2(want < (u64)2 * STBPE_PARTS ? (u64)2 * STBPE_PARTS : want);
    e->slots = slots;
    e->d.mask = slots - 1;
    // table slices: one per partition this rank can own (partitions with its residue modulo the
    // number of ranks), rounded up to a power of two
    const u64 slices = next_pow2(((u64)STBPE_PARTS + e->cfg.world_size - 1) / e->cfg.world_size);
    e->d.slot_bits = 0;
    while ((slices << e->d.slot_bits) < slots) ++e->d.slot_bits;
    // blocks of the arg-max over several ranks: at most 2^19
    e->d.blk_shift = 6;
    while ((slots >> e->d.blk_shift) > (1u << 19)) ++e->d.blk_shift;
    e->d.n_blocks = (unsigned int)(slots >> e->d.blk_shift);
}

// The device state, and the tied keys behind it, by way of pinned memory.  Synchronises the stream.
static int read_state(stbpe_engine *e, DevState *h, cudaStream_t s) {
    CK(cudaMemcpyAsync(e->pinned.p, e->d.st, STBPE_TIES_OFFSET + STBPE_TIES_CAP * sizeof(u64), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    memcpy(h, e->pinned.p, sizeof(DevState));
    return STBPE_OK;
}

static void drop_stream(stbpe_engine *e) {
    e->n_tokens = 0;
    e->d.n_tiles = 0;
    e->recs_stale = true;
    e->counted = false;
    e->only_bytes = true;
    e->filter_valid = false;
    e->wide_counted = e->full_refresh_pending = false;
    e->load_err = e->max_id = 0;
    e->bytes_below = e->made_below = 0;
    e->slots_needed = 0;
    e->merges_known = e->foreign_ids = false;
    e->state_stale = true;
}

// the device state of an empty stream, before the first work on it
static int fresh_state(stbpe_engine *e, cudaStream_t s) {
    if (!e->state_stale) return STBPE_OK;
    init_state_kernel<<<1, 1, 0, s>>>(e->d, e->cfg.base_vocab, 0);
    CK(cudaGetLastError());
    e->state_stale = false;
    return STBPE_OK;
}

STBPE_VISIBLE int stbpe_create(stbpe_engine **out, const stbpe_config *cfg) {
    if (!out || !cfg) return fail(nullptr, STBPE_E_BADARG, "null argument");
    if (cfg->max_tokens < 0 || cfg->max_merges < 0 || cfg->base_vocab < 0 || cfg->world_size < 1 ||
        cfg->rank < 0 || cfg->rank >= cfg->world_size)
        return fail(nullptr, STBPE_E_BADARG, "invalid configuration");
    if (cfg->max_tokens > 0x7FFFFFFFll * STBPE_TILE) return fail(nullptr, STBPE_E_BADARG, "max_tokens: tiles are numbered with 31 bits");
    if (cfg->world_size == 1 && cfg->table_slots > STBPE_MAX_SLOTS)
        return fail(nullptr, STBPE_E_BADARG, "table_slots: the candidate list holds 32-bit slot numbers");
    if ((i64)cfg->base_vocab + (i64)cfg->max_merges >= 0x7FFFFFFFll)
        return fail(nullptr, STBPE_E_ID_OVERFLOW, "Token id overflow: ids must stay below 2^31-1");
    stbpe_engine *e = new stbpe_engine();  // all members zero
    e->cfg = *cfg;
    e->dense32_min = -1;
    if (const char *v = getenv("STBPE_DENSE32_MIN_TOKENS")) e->dense32_min = atoll(v);
    e->narrow_counts = Best<uint16_t>::COUNTS;
    if (const char *v = getenv("STBPE_NARROW_COUNTS")) e->narrow_counts = atoll(v);
    e->use_graph = getenv("STBPE_NO_GRAPH") == nullptr;
    e->part_group = STBPE_PARTS;
    if (const char *v = getenv("STBPE_PART_GROUP")) e->part_group = atoi(v) > 0 ? atoi(v) : STBPE_PARTS;
    e->filter_density = 1.0;
    if (const char *v = getenv("STBPE_FILTER_DENSITY")) e->filter_density = atof(v);
    auto bail = [&](int code) {
        g_create_err = e->err;
        stbpe_destroy(e);
        return code;
    };
    cudaError_t c = cudaSetDevice(cfg->device);
    if (c != cudaSuccess) return bail(cuda_fail(e, c, "cudaSetDevice"));
    const DeviceInfo &info = device_info(cfg->device);
    if (info.err != cudaSuccess) return bail(cuda_fail(e, info.err, info.what));
    e->sm_count = info.sm_count;

    e->max_tokens = cfg->max_tokens;
    e->max_tiles = (int)((cfg->max_tokens + STBPE_TILE - 1) / STBPE_TILE);
    if (e->max_tiles < 1) e->max_tiles = 1;
    e->d.world = cfg->world_size;
    e->d.rank = cfg->rank;
    e->wide = starts_wide(*cfg);
    e->table_auto = cfg->table_slots <= 0 && cfg->world_size == 1;
    e->d.max_probe = e->table_auto ? STBPE_AUTO_PROBE : STBPE_MAX_PROBE;
    set_slots(e, cfg->table_slots > 0 ? (u64)cfg->table_slots : e->table_auto ? (u64)1 << 20 : auto_slots_mg(cfg->max_tokens));

#define ALLOC(ptr, n)                                                  \
    if ((c = dev_alloc(e, &(ptr), (size_t)(n))) != cudaSuccess) return bail(cuda_fail(e, c, "cudaMalloc " #ptr))
    {
        unsigned char *t = nullptr;
        e->tiles_bytes = (size_t)e->max_tiles * STBPE_TILE * tok_bytes(e);
        ALLOC(t, e->tiles_bytes);
        e->d.tiles = t;
    }
    {
        // everything small in one allocation; the pair table, the second stream buffer and the pair filter follow
        // when they are needed, in the size that is needed then
        Arena a;
        a.add(&e->d.recs, (size_t)e->max_tiles * 2);
        a.add(&e->d.tile_live, (size_t)e->max_tiles);
        a.add(&e->rp_lens, (size_t)e->max_tiles + 1);
        a.add(&e->rp_offs, (size_t)e->max_tiles + 1);
        cub::DeviceScan::ExclusiveSum(nullptr, e->rp_tmp_bytes, e->rp_lens, e->rp_offs, e->max_tiles + 1, 0);
        a.add((unsigned char **)&e->rp_tmp, e->rp_tmp_bytes ? e->rp_tmp_bytes : 16);
        a.add((unsigned char **)&e->d.st, STBPE_TIES_OFFSET + STBPE_TIES_CAP * sizeof(u64));  // state and tied keys: one copy
        a.add(&e->d.sync, 2);
        a.add(&e->d.merges, (size_t)2 * (cfg->max_merges + 1));
        a.add(&e->d.merge_counts, (size_t)cfg->max_merges + 1);
        a.add(&e->d.live_before, (size_t)cfg->max_merges + 1);
        a.add(&e->dense, 65536);
        a.add(&e->cand, 4);
        a.add(&e->all_cands, (size_t)4 * cfg->world_size);
        if (cfg->world_size > 1) {
            a.add(&e->d.blockmax, e->d.n_blocks);
            a.add(&e->d.dirty_bits, (e->d.n_blocks + 31) / 32);
            a.add(&e->partial, 4096);
        } else {
            a.add(&e->d.cand, STBPE_CAND_CAP);
            a.add(&e->d.cand_hist, STBPE_CAND_BUCKETS);
        }
        if ((c = a.alloc(e)) != cudaSuccess) return bail(cuda_fail(e, c, "cudaMalloc engine state"));
    }
    if (!e->table_auto) {
        ALLOC(e->d.table, e->slots);
        e->table_cap = e->slots;
    }
    c = stbpe::pinned_blocks().get(0, STBPE_PINNED_BYTES, &e->pinned);
    if (c != cudaSuccess) return bail(cuda_fail(e, c, "cudaMallocHost"));
    if (cfg->world_size > 1) {
        e->lslots = 1ull << 22;
        e->d.lmask = e->lslots - 1;
        e->d.cap_per_peer = 0;  // exchange buffers are set by stbpe_mg_set_buffers
        ALLOC(e->d.ltable, e->lslots);
        ALLOC(e->d.ltouched, 2 * e->lslots);
        c = cudaMemset(e->d.ltable, 0xFF, e->lslots * sizeof(Slot));
        if (c != cudaSuccess) return bail(cuda_fail(e, c, "cudaMemset ltable"));
        // counts of the local table must start at zero (keys at EMPTY = all ones)
        std::vector<Slot> init(1 << 16);
        for (auto &s : init) { s.key = STBPE_EMPTY; s.count = 0; }
        for (u64 off = 0; off < e->lslots; off += init.size()) {
            c = cudaMemcpy(e->d.ltable + off, init.data(), init.size() * sizeof(Slot), cudaMemcpyHostToDevice);
            if (c != cudaSuccess) return bail(cuda_fail(e, c, "cudaMemcpy ltable"));
        }
    }
#undef ALLOC
    c = e->d.dirty_bits ? cudaMemset(e->d.dirty_bits, 0, (e->d.n_blocks + 31) / 32 * sizeof(unsigned int))
                        : cudaMemset(e->d.cand_hist, 0, STBPE_CAND_BUCKETS * sizeof(unsigned int));
    if (c != cudaSuccess) return bail(cuda_fail(e, c, "cudaMemset"));

    e->count_smem = STBPE_COUNT_SMEM;
    e->select_grid = e->sm_count;
    e->refresh_grid = e->sm_count * 4;
    drop_stream(e);
    *out = e;
    return STBPE_OK;
}

STBPE_VISIBLE int stbpe_reset(stbpe_engine *e) {
    if (!e) return STBPE_E_BADARG;
    drop_stream(e);
    return STBPE_OK;
}

static int widen_stream(stbpe_engine *e, cudaStream_t s);

static int append_common(stbpe_engine *e, const void *data, i64 n, size_t elem, const i64 *row_offsets,
                         i64 n_rows, cudaStream_t s) {
    if (n < 0 || n_rows < 0 || (n > 0 && !data)) return fail(e, STBPE_E_BADARG, "bad append arguments");
    if (e->n_tokens + n > e->max_tokens)
        return fail(e, STBPE_E_CAPACITY, "token stream capacity exceeded");
    CK(cudaSetDevice(e->cfg.device));
    if (n == 0) return STBPE_OK;
    if (!e->recs_stale && e->n_tokens > 0) {
        // the stream has been counted: appending is still fine while no merge has rewritten a tile
        // (the tiles are dense and n_tokens is their true length), not afterwards
        DevState h;
        if (int rc_ = read_state(e, &h, s)) return rc_;
        if (h.merges_done > 0 || e->repacks_since_load > 0)
            return fail(e, STBPE_E_STATE, "rows cannot be appended after a merge has been applied; call stbpe_reset first");
    }
    const i64 single[2] = {0, n};
    const i64 *off = row_offsets ? row_offsets : single;
    const i64 rows = row_offsets ? n_rows : 1;
    if (off[0] != 0 || off[rows] != n) return fail(e, STBPE_E_BADARG, "row_offsets must start at 0 and end at n");
    if (int rc = fresh_state(e, s)) return rc;
    if (e->n_tokens == 0) {  // a fresh stream, into a buffer that takes all it may become (a re-pack may have left a smaller one)
        e->wide = starts_wide(e->cfg);
        const size_t full = (size_t)e->max_tiles * STBPE_TILE * tok_bytes(e);
        if (e->tiles_bytes < full && e->alt_bytes >= full) {
            std::swap(e->d.tiles, e->tiles_alt);
            std::swap(e->tiles_bytes, e->alt_bytes);
        }
        if (e->tiles_bytes < full) {
            dev_free(e, e->d.tiles);
            e->d.tiles = nullptr;
            e->tiles_bytes = 0;
            unsigned char *t = nullptr;
            CK(dev_alloc(e, &t, full));
            e->d.tiles = t;
            e->tiles_bytes = full;
        }
    }
    const i64 at0 = e->n_tokens;
    unsigned int *bad = &e->d.st->error;
    auto pack = [&](const void *src, i64 cnt, i64 at) {
        with_tok(e, [&](auto t) {
            typedef decltype(t) T;
            if (elem == 1) {
                i64 blocks = (cnt / 32 + 2 + 255) / 256;
                if (blocks > (i64)e->sm_count * 32) blocks = (i64)e->sm_count * 32;
                pack_bytes_kernel<T><<<(unsigned int)blocks, 256, 0, s>>>((const uint8_t *)src, cnt, e->d.tiles, at);
            } else {
                i64 blocks = (cnt / 16 + 255) / 256 + 1;
                if (blocks > (i64)e->sm_count * 8) blocks = (i64)e->sm_count * 8;
                pack_ids_kernel<T><<<(unsigned int)blocks, 256, 0, s>>>((const int32_t *)src, cnt, e->d.tiles, at, bad);
            }
        });
        return cudaGetLastError();
    };
    cudaPointerAttributes attr;
    if (cudaPointerGetAttributes(&attr, data) != cudaSuccess) {
        cudaGetLastError();
        attr.type = cudaMemoryTypeUnregistered;
    }
    const bool on_device = attr.type == cudaMemoryTypeDevice || attr.type == cudaMemoryTypeManaged;
    // The row offsets, and host data while they fit beside them, travel in one copy out of the engine's pinned
    // block; larger host data goes through a staging buffer in pieces, each packed as soon as it has landed.
    const size_t off_bytes = ((size_t)(rows + 1) * sizeof(i64) + 255) & ~(size_t)255, n_bytes = (size_t)n * elem;
    const size_t room = STBPE_PINNED_BYTES - STBPE_PINNED_STATE;
    const bool small = !on_device && off_bytes + n_bytes <= room;
    const size_t dev_bytes = off_bytes + (small ? n_bytes : 0);
    if (dev_bytes > e->off_cap) {
        dev_free(e, e->off_dev);
        e->off_dev = nullptr;
        e->off_cap = 0;
        unsigned char *t = nullptr;
        CK(dev_alloc(e, &t, dev_bytes));
        e->off_dev = t;
        e->off_cap = dev_bytes;
    }
    for (;;) {
        if (off_bytes <= room) {
            char *pin = (char *)e->pinned.p + STBPE_PINNED_STATE;
            memcpy(pin, off, (size_t)(rows + 1) * sizeof(i64));
            if (small) memcpy(pin + off_bytes, data, n_bytes);
            CK(cudaMemcpyAsync(e->off_dev, pin, dev_bytes, cudaMemcpyHostToDevice, s));
        } else {
            CK(cudaMemcpyAsync(e->off_dev, off, (size_t)(rows + 1) * sizeof(i64), cudaMemcpyHostToDevice, s));
        }
        if (on_device) {
            CK(pack(data, n, at0));
        } else if (small) {
            CK(pack((char *)e->off_dev + off_bytes, n, at0));
        } else {
            const size_t half = n_bytes < ((size_t)32 << 20) ? ((n_bytes + 255) & ~(size_t)255) : (size_t)32 << 20;
            unsigned char *stage = nullptr;
            CK(dev_alloc(e, &stage, 2 * half));
            const cudaError_t c = stbpe::staged_copy(data, (size_t)n, elem, attr.type == cudaMemoryTypeUnregistered, stage, half, s,
                                                     [&](void *src, size_t at, size_t cnt) { return pack(src, (i64)cnt, at0 + (i64)at); });
            const cudaError_t c2 = cudaStreamSynchronize(s);
            dev_free(e, stage);
            CK(c);
            CK(c2);
        }
        with_tok(e, [&](auto t) {
            mark_row_starts_kernel<decltype(t)><<<(unsigned int)((rows + 255) / 256), 256, 0, s>>>((const i64 *)e->off_dev, rows, e->d.tiles, at0);
        });
        CK(cudaGetLastError());
        // the host offsets (and a host source) must stay valid until the copies ran
        if (elem == 1) {
            CK(cudaStreamSynchronize(s));
            break;
        }
        unsigned int *err = (unsigned int *)e->pinned.p;  // error bits and the largest id behind them
        CK(cudaMemcpyAsync(err, bad, 2 * sizeof(*err), cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        if (err[1] > e->max_id) e->max_id = err[1];
        e->load_err |= *err & ~STBPE_DERR_NARROW;
        if (!(*err & STBPE_DERR_NARROW)) break;
        // an id that 15 bits cannot hold: what the stream holds so far is widened, and this piece is packed again
        *err &= ~STBPE_DERR_NARROW;
        CK(cudaMemcpyAsync(bad, err, sizeof(*err), cudaMemcpyHostToDevice, s));
        int rc = widen_stream(e, s);
        if (rc != STBPE_OK) return rc;
    }
    e->n_tokens += n;
    e->recs_stale = true;
    e->counted = false;
    if (elem == 1)
        e->bytes_below = 256;
    else
        e->only_bytes = false;
    return STBPE_OK;
}

// Rows of a padded host batch one behind the other, as bytes (elem 1) or ids (elem 4).  One pass over the batch; the
// same in tensor operations (sum, comparison with a prefix, boolean gather, cast) took five.
STBPE_VISIBLE int stbpe_flatten_rows(const int32_t *tokens, const uint8_t *valid, int64_t rows, int64_t width, int32_t elem, void *out,
                                     int64_t *lengths) {
    if (rows < 0 || width < 0 || (elem != 1 && elem != 4) || (rows > 0 && (!lengths || (width > 0 && (!tokens || !valid || !out))))) return STBPE_E_BADARG;
    unsigned char *to = (unsigned char *)out;
    for (i64 r = 0; r < rows; ++r, tokens += width, valid += width) {
        const void *end = width > 0 ? memchr(valid, 0, (size_t)width) : nullptr;
        const i64 n = end ? (const uint8_t *)end - valid : width;
        uint8_t later = 0;
        for (i64 i = n; i < width; ++i) later |= valid[i];
        if (later) return STBPE_E_STATE;
        lengths[r] = n;
        if (elem == 4) {
            if (n) memcpy(to, tokens, (size_t)n * 4);
        } else {
            uint32_t seen = 0;
            for (i64 i = 0; i < n; ++i) {
                seen |= (uint32_t)tokens[i];
                to[i] = (unsigned char)tokens[i];
            }
            if (seen > 255u) return STBPE_E_ID_OVERFLOW;
        }
        to += n * elem;
    }
    return STBPE_OK;
}

STBPE_VISIBLE int stbpe_append_bytes(stbpe_engine *e, const uint8_t *data, int64_t n,
                                     const int64_t *row_offsets, int64_t n_rows, void *stream) {
    if (!e) return STBPE_E_BADARG;
    return append_common(e, data, n, 1, (const i64 *)row_offsets, n_rows, (cudaStream_t)stream);
}

STBPE_VISIBLE int stbpe_append_ids(stbpe_engine *e, const int32_t *ids, int64_t n,
                                   const int64_t *row_offsets, int64_t n_rows, void *stream) {
    if (!e) return STBPE_E_BADARG;
    return append_common(e, ids, n, 4, (const i64 *)row_offsets, n_rows, (cudaStream_t)stream);
}

static int check_error_bits(stbpe_engine *e, unsigned int err) {
    if (err & STBPE_DERR_BAD_ID)
        return fail(e, STBPE_E_ID_OVERFLOW, "Token id overflow: ids must be in [0, 2^31-2]");
    if (err & STBPE_DERR_TABLE_FULL)
        return fail(e, STBPE_E_CAPACITY, "pair workspace capacity exceeded (pair table full: create the engine with more table_slots, GPUBPETrainer.table_slots)");
    if (err & STBPE_DERR_OUTBOX_FULL) return fail(e, STBPE_E_CAPACITY, "pair workspace capacity exceeded (delta outbox full)");
    if (err & STBPE_DERR_LTABLE_FULL) return fail(e, STBPE_E_CAPACITY, "pair workspace capacity exceeded (local delta table full)");
    if (err & STBPE_DERR_TIMEOUT) return fail(e, STBPE_E_TIMEOUT, "a bounded device-side wait gave up (tile pipeline or a peer's flag)");
    if (err & STBPE_DERR_KEY_MISSING) return fail(e, STBPE_E_STATE, "selected pair missing from the pair table");
    return STBPE_OK;
}

static int check_device_error(stbpe_engine *e, cudaStream_t s, unsigned int *bits = nullptr) {
    unsigned int err = 0;
    CK(cudaMemcpyAsync(&err, &e->d.st->error, sizeof(err), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    if (bits) *bits = err;
    return check_error_bits(e, err);
}

static int prepare_stream_state(stbpe_engine *e, cudaStream_t s) {
    if (e->recs_stale) {
        int rc = check_error_bits(e, e->load_err);  // id range flag from the pack kernels
        if (rc != STBPE_OK) return rc;
        e->d.n_tiles = (int)((e->n_tokens + STBPE_TILE - 1) / STBPE_TILE);
        if (e->d.n_tiles > 0) {
            with_tok(e, [&](auto t) {
                init_recs_kernel<decltype(t)><<<(e->d.n_tiles + 255) / 256, 256, 0, s>>>(e->d, e->n_tokens);
            });
            CK(cudaGetLastError());
        }
        init_state_kernel<<<1, 1, 0, s>>>(e->d, e->cfg.base_vocab, e->n_tokens);
        CK(cudaGetLastError());
        e->state_stale = false;
        e->merges_done = 0;
        e->merges_known = true;
        e->recs_stale = false;
        e->repacks_since_load = 0;
        e->filter_valid = false;  // a fresh stream starts without a pair filter (see filter_policy)
    }
    return STBPE_OK;
}

__global__ void clear_skip_state_kernel(EngineDev e, int valid) {
    e.st->n_work = 0;  // a merge that is committed but not yet applied counts its tiles from here
    e.st->filter_valid = valid;
}

// The pair filter follows the tile layout: it is rebuilt from the stream, or declared stale.
static int rebuild_presence(stbpe_engine *e, cudaStream_t s) {
    const size_t groups = ((size_t)e->d.n_tiles + 31) / 32;
    if (groups > e->presence_cap) {
        CK(cudaStreamSynchronize(s));
        dev_free(e, e->d.presence);
        e->d.presence = nullptr;
        e->presence_cap = 0;
        CK(dev_alloc(e, &e->d.presence, (size_t)STBPE_PPITCH * groups));
        e->presence_cap = groups;
    }
    clear_skip_state_kernel<<<1, 1, 0, s>>>(e->d, 1);
    CK(cudaGetLastError());
    e->filter_valid = true;
    if (e->d.n_tiles > 0) {
        with_tok(e, [&](auto t) {
            presence_rebuild_kernel<decltype(t)><<<e->sm_count * 2, 1024, STBPE_PROWS * sizeof(unsigned int), s>>>(e->d);
        });
        CK(cudaGetLastError());
    }
    return STBPE_OK;
}

// Buffers of the partitioned first count (wide_count.cuh), one allocation: every CTA of the first
// pass owns a region of every partition, sized for its share of the partition's words (1 / grid of
// them, give or take the statistics of its batches) plus head room.
static int wide_alloc(stbpe_engine *e) {
    if (e->wide_block) return STBPE_OK;
    const int n_cta = e->sm_count;
    const i64 cap = ((e->max_tokens / STBPE_PARTS / n_cta) * 13 / 10 + 1024 + 3) & ~(i64)3;
    const size_t bytes = STBPE_WIDE_HEADER_BYTES + wide_fill_bytes(n_cta) + 65536 * sizeof(u64) +
                         (size_t)STBPE_PARTS * n_cta * cap * sizeof(uint32_t);
    size_t free_b = 0, total_b = 0;
    CK(cudaMemGetInfo(&free_b, &total_b));
    if (free_b < bytes + ((size_t)2 << 30)) return fail(e, STBPE_E_CAPACITY, "CUDA out of memory (pair partitions)");
    cudaError_t c = dev_alloc(e, &e->wide_block, bytes);
    if (c != cudaSuccess) return cuda_fail(e, c, "cudaMalloc pair partitions");
    WideHeader hd;
    hd.cap = cap;
    hd.n_cta = n_cta;
    CK(cudaMemcpy(e->wide_block, &hd, sizeof(hd), cudaMemcpyHostToDevice));
    e->parts.fill = const_cast<unsigned int *>(wide_fill(e->wide_block));
    e->wide_dense = const_cast<u64 *>(wide_dense(e->wide_block, n_cta));
    e->parts.words = const_cast<uint32_t *>(wide_words(e->wide_block, n_cta));
    e->parts.cap = cap;
    e->parts.n_cta = n_cta;
    return STBPE_OK;
}

// the pair table has `want` slots; its memory is kept while it is large enough
static int set_table(stbpe_engine *e, u64 want) {
    set_slots(e, want);
    if (e->d.table && e->table_cap >= e->slots) return STBPE_OK;
    dev_free(e, e->d.table);
    e->d.table = nullptr;
    e->table_cap = 0;
    cudaError_t c = dev_alloc(e, &e->d.table, e->slots);
    if (c != cudaSuccess) return cuda_fail(e, c, "cudaMalloc pair table");
    e->table_cap = e->slots;
    return STBPE_OK;
}

// Four times the slots: the keys that still have a count move over.  Slots change, so the candidate list ends.
static int grow_table(stbpe_engine *e, cudaStream_t s) {
    Slot *old = e->d.table;
    const u64 old_slots = e->slots;
    Slot *fresh = nullptr;
    cudaError_t c = old_slots * 4 > (u64)STBPE_MAX_SLOTS ? cudaErrorMemoryAllocation : dev_alloc(e, &fresh, old_slots * 4);
    if (c != cudaSuccess) {
        cudaGetLastError();
        e->table_auto = false;  // no room: go on in the table there is, a full one is an error status
        e->d.max_probe = STBPE_MAX_PROBE;
        return STBPE_OK;
    }
    set_slots(e, old_slots * 4);
    e->d.table = fresh;
    e->table_cap = e->slots;
    clear_table_kernel<<<e->sm_count * 8, 256, 0, s>>>(e->d);
    cand_none_kernel<<<1, 1, 0, s>>>(e->d);
    e->cand_stale = true;
    CK(cudaMemsetAsync(&e->d.st->n_keys, 0, sizeof(u64), s));
    rehash_kernel<<<e->sm_count * 8, 256, 0, s>>>(e->d, old, old_slots);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(s));
    dev_free(e, old);
    return STBPE_OK;
}

// what every count starts with: tile records of a fresh stream, an empty table, no maxima
static int count_prologue(stbpe_engine *e, bool clear, cudaStream_t s) {
    const bool fresh = e->recs_stale;
    e->convert_ms = e->count_ms = 0.f;
    e->count_timed = false;
    int rc = prepare_stream_state(e, s);
    if (rc != STBPE_OK) return rc;
    if (e->table_auto) {
        // A stream of bytes starts with at most 65 536 pairs and its table grows with the keys (grow_table): a table
        // of 16 MB stays in L2 and costs nothing to clear or scan, one for every pair a run might create is
        // half a gigabyte on 128 MB of text.  Other streams may hold any number of pairs from the start.
        u64 want = std::max(e->only_bytes ? (u64)1 << 20 : auto_slots(e->n_tokens, ids_below(e)), e->slots_needed);
        if (!fresh && e->slots > want) want = e->slots;  // a recount of the rewritten stream
        rc = set_table(e, want);
        if (rc != STBPE_OK) return rc;
    }
    if (clear) clear_table_kernel<<<e->sm_count * 8, 256, 0, s>>>(e->d);
    CK(cudaGetLastError());
    if (e->cfg.world_size > 1) {
        CK(cudaMemsetAsync(e->d.dirty_bits, 0, (e->d.n_blocks + 31) / 32 * sizeof(unsigned int), s));
        CK(cudaMemsetAsync(e->d.blockmax, 0, (size_t)e->d.n_blocks * sizeof(Slot), s));  // count 0 = no candidate
    } else {
        cand_none_kernel<<<1, 1, 0, s>>>(e->d);
    e->cand_stale = true;
        CK(cudaGetLastError());
    }
    CK(cudaMemsetAsync(&e->d.st->n_keys, 0, sizeof(u64), s));
    if (!e->ev0) {
        CK(cudaEventCreate(&e->ev0));
        CK(cudaEventCreate(&e->ev1));
    }
    return STBPE_OK;
}

// Whether the partitioned count takes a stream: fresh, ids below 65 536, and long enough for its fixed 0.4 ms (six launches, two
// reads of the error bits).  What the general kernel takes depends on how many pairs are distinct, that is on the ids: over
// 65 536 ids, general / partitioned on an engine that has counted before, 2^19 0.44 / 0.45 ms, 2^20 0.57 / 0.48, 2^21 0.84 /
// 0.50, 2^22 1.45 / 0.54, 2^24 4.3 / 0.68; over 4 096, 2^20 0.38 / 0.47, 2^21 0.52 / 0.49, 2^22 1.01 / 0.56; over 512, 2^22
// 0.37 / 0.48, 2^23 0.61 / 0.51, 2^24 1.15 / 0.55.  A new engine pays 0.1 ms more for the partition buffers: 2^21 0.85 / 0.64,
// 0.52 / 0.61 and 0.28 / 0.61, 2^23 over 512 ids 0.63 / 0.63.
static bool wide_eligible(const stbpe_engine *e, bool fresh) {
    const i64 ids = ids_below(e), least = e->dense32_min >= 0 ? e->dense32_min : ids >= 4096 ? 1ll << 21 : 1ll << 23;
    return e->n_tokens > 0 && e->n_tokens < (1ll << 32) && e->slots <= (1ull << 30) && fresh && !e->only_bytes && e->cfg.base_vocab <= 65536 &&
           ids <= 65536 && e->n_tokens >= least && !getenv("STBPE_NO_DENSE_COUNT");
}

// first pass of the partitioned count; *ok = 0 when an id of 65 536 or more or a full region made it give up
static int wide_pass1(stbpe_engine *e, int *ok, cudaStream_t s) {
    PartBuffers &pb = e->parts;
    *ok = 0;
    CK(cudaMemsetAsync(e->wide_dense, 0, 65536 * sizeof(u64), s));
    CK(cudaEventRecord(e->ev0, s));
    with_tok(e, [&](auto t) {
        partition_pairs_kernel<decltype(t)><<<pb.n_cta, STBPE_PART_THREADS, STBPE_PART_SMEM_BYTES, s>>>(e->d, e->wide_dense, pb);
    });
    CK(cudaGetLastError());
    CK(cudaEventRecord(e->ev1, s));
    unsigned int derr = 0;
    CK(cudaMemcpyAsync(&derr, &e->d.st->error, sizeof(derr), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    CK(cudaEventElapsedTime(&e->count_ms, e->ev0, e->ev1));
    if (derr & STBPE_DERR_DENSE_OVERFLOW) {
        derr &= ~STBPE_DERR_DENSE_OVERFLOW;
        CK(cudaMemcpyAsync(&e->d.st->error, &derr, sizeof(derr), cudaMemcpyHostToDevice, s));
        CK(cudaStreamSynchronize(s));
        return STBPE_OK;
    }
    *ok = 1;
    return STBPE_OK;
}

// From here on the partitions' words are added to a cleared table one by one, as several ranks do it, instead of
// being ordered and built range by range.  2^30 slots: the ranges outgrow the 64 KB of shared memory that let three
// CTAs share an SM (2.5e8 ids 7.3 instead of 8.8 ms, 2^30 ids 16.7 instead of 25.9).  2^29 slots: 256 ranges per
// partition leave a piece few words of each, while the adds of a partition stay inside 32 MB of L2 and the longer
// a region, the more of them the word caches take.  Ordered / one by one, whole count in ms: 2^30 ids 14.8 / 15.4, 1.4e9
// 17.7 / 17.7, 1.7e9 21.3 / 20.0, 2^31 25.6 / 24.1, 2.8e9 31.7 / 30.4 (ids below 4 096: 1.4e9 12.3 / 13.1, 1.7e9 15.6 / 14.7).
// Smaller tables: 2^28 slots and 1.7e9 ids 19.2 / 21.4.
static bool wide_one_by_one(const stbpe_engine *e) {
    return e->slots > (1ull << 29) || (e->slots == (1ull << 29) && e->n_tokens >= 3ll << 29);
}

// second and third pass of the partitioned count; *ok = 0 when the spill list ran over
static int wide_build(stbpe_engine *e, int *ok, cudaStream_t s) {
    const PartBuffers &pb = e->parts;
    if (wide_one_by_one(e)) {
        WidePeers own = {};
        own.block[0] = e->wide_block;
        own.world = 1;
        CK(cudaEventRecord(e->ev0, s));
        clear_table_kernel<<<e->sm_count * 8, 256, 0, s>>>(e->d);
        dense_to_table_kernel<false><<<256, 256, 0, s>>>(e->d, e->wide_dense);
        partition_table_peers_kernel<<<pb.n_cta * 2 * STBPE_PARTS, 1024, 0, s>>>(e->d, own, 0, 1, pb.n_cta);
        CK(cudaGetLastError());
        CK(cudaEventRecord(e->ev1, s));
        CK(cudaEventSynchronize(e->ev1));
        CK(cudaEventElapsedTime(&e->convert_ms, e->ev0, e->ev1));
        e->count_ms += e->convert_ms;
        *ok = 1;
        return STBPE_OK;
    }
    int lg = 0;
    while ((1ull << lg) < e->slots) ++lg;
    // ranges of 2^13 slots: 64 KB of shared memory, three CTAs per SM; at least one bit and at most eight bits of
    // ordering, so small tables get smaller ranges
    const int task_bits = lg - STBPE_PART_BITS - 1 < 13 ? lg - STBPE_PART_BITS - 1 : 13;
    const int sub_bits = lg - STBPE_PART_BITS - task_bits;
    const int chunk = sub_bits > 6 ? 16384 : 8192;
    const int cpr = (int)((pb.cap + chunk - 1) / chunk);
    const i64 n_chunks = (i64)STBPE_PARTS * pb.n_cta * cpr;
    const unsigned int spill_cap = 1u << 20;
    const size_t offs_bytes = ((size_t)n_chunks * ((1 << sub_bits) + 1) * sizeof(uint16_t) + 255) & ~(size_t)255;
    unsigned char *scratch = nullptr;
    CK(dev_alloc(e, &scratch, offs_bytes + (size_t)spill_cap * sizeof(uint32_t) + 256));
    uint16_t *offs = (uint16_t *)scratch;
    unsigned int *n_spill = (unsigned int *)(scratch + offs_bytes);
    uint32_t *spill = (uint32_t *)(scratch + offs_bytes + 256);
    const size_t build_smem = (size_t)8 << task_bits;
    CK(cudaEventRecord(e->ev0, s));
    CK(cudaMemsetAsync(n_spill, 0, sizeof(*n_spill), s));
    if (chunk == 8192)
        sub_partition_kernel<8192><<<e->sm_count * 3, STBPE_SUB_THREADS, 8192 * sizeof(uint32_t), s>>>(pb, cpr, sub_bits, offs);
    else
        sub_partition_kernel<16384><<<e->sm_count * 2, STBPE_SUB_THREADS, 16384 * sizeof(uint32_t), s>>>(pb, cpr, sub_bits, offs);
    build_table_kernel<<<e->sm_count * 3, STBPE_BUILD_THREADS, build_smem, s>>>(e->d, pb, chunk, cpr, sub_bits, task_bits, offs, spill, n_spill, spill_cap);
    spill_to_table_kernel<<<e->sm_count, 256, 0, s>>>(e->d, spill, n_spill, spill_cap);
    dense_to_table_kernel<false><<<256, 256, 0, s>>>(e->d, e->wide_dense);
    CK(cudaGetLastError());
    CK(cudaEventRecord(e->ev1, s));
    unsigned int *derr = (unsigned int *)e->pinned.p;
    CK(cudaMemcpyAsync(derr, &e->d.st->error, sizeof(*derr), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    dev_free(e, scratch);
    CK(cudaEventElapsedTime(&e->convert_ms, e->ev0, e->ev1));
    e->count_ms += e->convert_ms;  // the pair table is complete only after all passes
    *ok = (*derr & STBPE_DERR_DENSE_OVERFLOW) == 0;
    if (!*ok) {
        *derr &= ~STBPE_DERR_DENSE_OVERFLOW;
        CK(cudaMemcpyAsync(&e->d.st->error, derr, sizeof(*derr), cudaMemcpyHostToDevice, s));
        CK(cudaStreamSynchronize(s));
    }
    return STBPE_OK;
}

// *err: the device error bits, where they have been read behind the last kernel (*err_known).
static int launch_count(stbpe_engine *e, bool mg, cudaStream_t s, unsigned int *err = nullptr, bool *err_known = nullptr) {
    if (mg && e->wide_counted) {  // stbpe_mg_wide_pass2 has filled the table already
        e->wide_counted = false;
        return STBPE_OK;
    }
    const bool fresh = e->recs_stale, wide = !mg && wide_eligible(e, fresh);
    int rc = count_prologue(e, !wide, s);  // the partitioned count writes or clears every slot of the table itself
    if (rc != STBPE_OK) return rc;
    if (e->d.n_tiles > 0 && fresh && e->only_bytes && !getenv("STBPE_NO_DENSE_COUNT")) {
        // byte-level fast path: dense stream, ids < 256
        CK(cudaMemsetAsync(e->dense, 0, 65536 * sizeof(u64), s));
        CK(cudaEventRecord(e->ev0, s));
        with_tok(e, [&](auto t) {
            count_dense_kernel<decltype(t)><<<e->sm_count, STBPE_DENSE_THREADS, 32768 * 4, s>>>(e->d, e->dense);
        });
        CK(cudaGetLastError());
        // one rank: into the table at once, an overflow is looked at with the final error check and counts again;
        // several ranks: the deltas of a failed count must not reach the rank-local table
        if (!mg) dense_to_table_kernel<false><<<256, 256, 0, s>>>(e->d, e->dense);
        CK(cudaGetLastError());
        CK(cudaEventRecord(e->ev1, s));
        e->count_timed = true;
        unsigned int *derr = (unsigned int *)e->pinned.p;  // error bits and the largest id behind them
        CK(cudaMemcpyAsync(derr, &e->d.st->error, 2 * sizeof(*derr), cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        if (!(*derr & STBPE_DERR_DENSE_OVERFLOW)) {
            if (!mg) e->bytes_below = (i64)derr[1] + 1;
            if (!mg && err) *err = *derr, *err_known = true;
            if (mg) dense_to_table_kernel<true><<<256, 256, 0, s>>>(e->d, e->dense);
            CK(cudaGetLastError());
            return STBPE_OK;
        }
        // a 16-bit counter came too close to its limit: discard and count with the general kernel
        *derr &= ~STBPE_DERR_DENSE_OVERFLOW;
        CK(cudaMemcpyAsync(&e->d.st->error, derr, sizeof(*derr), cudaMemcpyHostToDevice, s));
        CK(cudaStreamSynchronize(s));
        rc = count_prologue(e, true, s);
        if (rc != STBPE_OK) return rc;
    }
    if (wide) {
        // 16-bit vocabulary: partition the pairs, order them inside their partitions and build the table range
        // by range (wide_count.cuh).  The partition buffers are allocated at first use and kept for later counts;
        // without room for them the general kernel counts.
        int ok = 0;
        if (wide_alloc(e) == STBPE_OK) {
            rc = wide_pass1(e, &ok, s);
            if (rc != STBPE_OK) return rc;
        }
        if (ok) {
            rc = wide_build(e, &ok, s);
            if (rc != STBPE_OK) return rc;
            if (ok) return STBPE_OK;
        }
        clear_table_kernel<<<e->sm_count * 8, 256, 0, s>>>(e->d);
        CK(cudaMemsetAsync(&e->d.st->n_keys, 0, sizeof(u64), s));
        // an id of 65 536 or more, or a region outgrew its buffer: the general kernel counts
    }
    if (e->d.n_tiles > 0) {
        const int warps = STBPE_COUNT_THREADS / 32, need = (e->d.n_tiles + warps - 1) / warps;
        const int grid = need < 2 * e->sm_count ? need : 2 * e->sm_count;
        CK(cudaEventRecord(e->ev0, s));
        with_tok(e, [&](auto t) {
            typedef decltype(t) T;
            if (mg)
                count_kernel<T, true><<<grid, STBPE_COUNT_THREADS, e->count_smem, s>>>(e->d);
            else
                count_kernel<T, false><<<grid, STBPE_COUNT_THREADS, e->count_smem, s>>>(e->d);
        });
        CK(cudaGetLastError());
        CK(cudaEventRecord(e->ev1, s));
        e->count_timed = true;
    }
    return STBPE_OK;
}

static int launch_refresh(stbpe_engine *e, int all, cudaStream_t s) {
    refresh_kernel<<<e->refresh_grid, 256, 0, s>>>(e->d, all);
    CK(cudaGetLastError());
    return STBPE_OK;
}

STBPE_VISIBLE int stbpe_count_initial(stbpe_engine *e, void *stream) {
    if (!e) return STBPE_E_BADARG;
    cudaStream_t s = (cudaStream_t)stream;
    CK(cudaSetDevice(e->cfg.device));
    if (e->cfg.world_size > 1) return fail(e, STBPE_E_STATE, "use stbpe_mg_count_local on a multi-rank engine");
    e->counted = false;  // (a recount that finds no memory for a larger table leaves none)
    for (;;) {
        const bool fresh = e->recs_stale;
        unsigned int err = 0;
        bool err_known = false;
        int rc = launch_count(e, false, s, &err, &err_known);
        if (rc != STBPE_OK) return rc;
        rc = err_known ? check_error_bits(e, err) : check_device_error(e, s, &err);
        if ((err & STBPE_DERR_TABLE_FULL) && e->table_auto && e->slots * 4 <= (u64)STBPE_MAX_SLOTS) {
            // more distinct pairs than the table was sized for: the same count once more, with four times the slots
            e->slots_needed = e->slots * 4;
            e->recs_stale = fresh;
            CK(cudaMemsetAsync(&e->d.st->error, 0, sizeof(err), s));
            continue;
        }
        e->counted = true;
        return rc;
    }
}

// Candidate list of the pair table as it stands: threshold search (one pass over the table in the usual case,
// further ones while a bucket holds too many pairs), then the list.
static int queue_refill(stbpe_engine *e, cudaStream_t s) {
    const u64 key_hi = e->wide ? 0x7FFFFFFFFFFFFFFFull : ((u64)Tok<uint16_t>::IDMASK << 32) | Tok<uint16_t>::IDMASK;
    const i64 want = ((i64)e->slots + 511) / 512;
    const unsigned int grid = (unsigned int)(want < e->sm_count * 4 ? want : e->sm_count * 4);
    cand_hist_kernel<<<grid, 512, 0, s>>>(e->d);
    cand_decide_kernel<<<1, 1024, 0, s>>>(e->d, key_hi);
    cand_collect_kernel<<<grid, 512, 0, s>>>(e->d);
    CK(cudaGetLastError());
    return STBPE_OK;
}
static int refill_candidates(stbpe_engine *e, cudaStream_t s) {
    CK(cudaMemsetAsync(&e->d.st->cand_state, 0, sizeof(int), s));
    for (int pass = 0; pass < 16; ++pass) {
        if (int rc_ = queue_refill(e, s)) return rc_;
        DevState h;
        if (int rc_ = read_state(e, &h, s)) return rc_;
        if (h.cand_state == STBPE_CAND_READY) {
            e->cand_stale = false;
            return STBPE_OK;
        }
    }
    return fail(e, STBPE_E_STATE, "no candidate threshold found");
}

// The best count and the keys that hold it, ascending, out of the candidate list (or out of a scan of the table
// when the list does not hold all of them).  `queued`: the kernel has run behind a merge and was read with it.
static int tied_candidates(stbpe_engine *e, bool queued, std::vector<u64> *keys, i64 *count, cudaStream_t s) {
    keys->clear();
    for (int attempt = 0; attempt < 2; ++attempt) {
        DevState h;
        if (queued) {
            memcpy(&h, e->pinned.p, sizeof(h));
        } else {
            ties_kernel<<<1, 1024, 0, s>>>(e->d);
            CK(cudaGetLastError());
            if (int rc = read_state(e, &h, s)) return rc;
        }
        queued = false;
        if (!h.peek_valid) {
            int rc = refill_candidates(e, s);
            if (rc != STBPE_OK) return rc;
            continue;
        }
        *count = h.peek_count;
        if (h.peek_count <= 0) return STBPE_OK;
        if (h.peek_ties > 0 && h.peek_ties <= STBPE_TIES_CAP) {
            const u64 *k = (const u64 *)((const char *)e->pinned.p + STBPE_TIES_OFFSET);
            keys->assign(k, k + h.peek_ties);
        } else {
            CK(cudaMemsetAsync(&e->d.st->peek_ties, 0, sizeof(i64), s));
            count_ties_kernel<<<e->sm_count * 8, 256, 0, s>>>(e->d);
            CK(cudaGetLastError());
            DevState h2;
            if (int rc = read_state(e, &h2, s)) return rc;
            stbpe::Block b;
            CK(stbpe::device_blocks().get(e->cfg.device, (size_t)h2.peek_ties * sizeof(u64), &b));
            CK(cudaMemsetAsync(&e->d.st->export_n, 0, sizeof(i64), s));
            export_ties_kernel<<<e->sm_count * 8, 256, 0, s>>>(e->d, h.peek_count, (u64 *)b.p, h2.peek_ties);
            CK(cudaGetLastError());
            keys->resize((size_t)h2.peek_ties);
            CK(cudaMemcpyAsync(keys->data(), b.p, keys->size() * sizeof(u64), cudaMemcpyDeviceToHost, s));
            CK(cudaStreamSynchronize(s));
            stbpe::device_blocks().put(e->cfg.device, b);
        }
        std::sort(keys->begin(), keys->end());
        keys->erase(std::unique(keys->begin(), keys->end()), keys->end());  // a candidate may be listed twice
        return STBPE_OK;
    }
    return fail(e, STBPE_E_STATE, "no candidate found");
}

// Best pair of the table into the device state, or as the loop's next step; *h = the state afterwards.
static int choose(stbpe_engine *e, bool advance, DevState *h, cudaStream_t s) {
    for (int attempt = 0; attempt < 2; ++attempt) {
        choose_kernel<<<1, 1024, 0, s>>>(e->d, advance ? 1 : 0);
        CK(cudaGetLastError());
        if (int rc_ = read_state(e, h, s)) return rc_;
        if (h->peek_valid || (advance && h->stopped)) return STBPE_OK;
        int rc = refill_candidates(e, s);
        if (rc != STBPE_OK) return rc;
    }
    return fail(e, STBPE_E_STATE, "no candidate found");
}

STBPE_VISIBLE int stbpe_select_best(stbpe_engine *e, uint64_t *key, int64_t *count, int64_t *n_ties,
                                    void *stream) {
    if (!e || !key || !count) return STBPE_E_BADARG;
    cudaStream_t s = (cudaStream_t)stream;
    CK(cudaSetDevice(e->cfg.device));
    if (!e->counted) return fail(e, STBPE_E_STATE, "count the pairs before selecting");
    DevState h;
    if (e->cfg.world_size > 1) {
        select_kernel<<<e->select_grid, STBPE_SELECT_THREADS, 0, s>>>(e->d, 0, e->partial, e->cand);
        CK(cudaGetLastError());
    } else {
        int rc = choose(e, false, &h, s);
        if (rc != STBPE_OK) return rc;
    }
    if (n_ties) {
        CK(cudaMemsetAsync(&e->d.st->peek_ties, 0, sizeof(i64), s));
        count_ties_kernel<<<e->sm_count * 8, 256, 0, s>>>(e->d);
        CK(cudaGetLastError());
    }
    if (int rc_ = read_state(e, &h, s)) return rc_;
    *key = h.peek_count > 0 ? h.peek_key : 0;
    *count = h.peek_count;
    if (n_ties) *n_ties = h.peek_count > 0 ? h.peek_ties : 0;
    return STBPE_OK;
}

static int filter_policy(stbpe_engine *e, const DevState &h, bool layout_changed, cudaStream_t s);
struct Draws {  // outputs of a tie-breaking generator on the device
    const uint32_t *dev;
    int n, used;
};
static int run_forced(stbpe_engine *e, const int32_t *pairs, int n, int32_t first_new, int64_t *n_matches, cudaStream_t s, bool then_ties = false,
                      int most = 0, int *n_done = nullptr, Draws *draws = nullptr);

static int launch_merge(stbpe_engine *e, bool mg, cudaStream_t s) {
    if (e->d.n_tiles < 1) return STBPE_OK;
    with_tok(e, [&](auto t) {
        typedef decltype(t) T;
        if (mg)
            merge_kernel<T, true><<<e->sm_count, MergeGeom<T>::THREADS, MergeGeom<T>::BYTES, s>>>(e->d, unit_shift(e, e->sm_count));
        else
            merge_kernel<T, false><<<e->sm_count, MergeGeom<T>::THREADS, MergeGeom<T>::BYTES, s>>>(e->d, unit_shift(e, e->sm_count));
    });
    CK(cudaGetLastError());
    return STBPE_OK;
}

STBPE_VISIBLE int stbpe_apply_merge(stbpe_engine *e, int32_t a, int32_t b, int32_t new_id,
                                    int64_t *n_matches, void *stream) {
    if (!e) return STBPE_E_BADARG;
    cudaStream_t s = (cudaStream_t)stream;
    CK(cudaSetDevice(e->cfg.device));
    if (!e->counted) return fail(e, STBPE_E_STATE, "count the pairs before merging");
    if (e->cfg.world_size > 1) return fail(e, STBPE_E_STATE, "single-rank entry point");
    if (a < 0 || b < 0 || new_id < 0 || a == 0x7FFFFFFF || b == 0x7FFFFFFF || new_id == 0x7FFFFFFF)
        return fail(e, STBPE_E_ID_OVERFLOW, "Token id overflow: ids must be in [0, 2^31-2]");
    const int32_t pair[2] = {a, b};
    return run_forced(e, pair, 1, new_id, n_matches, s);
}

STBPE_VISIBLE int stbpe_apply_merges(stbpe_engine *e, const int32_t *pairs, int32_t n, int32_t first_new_id, void *stream) {
    if (!e || n < 0 || (n > 0 && !pairs)) return STBPE_E_BADARG;
    CK(cudaSetDevice(e->cfg.device));
    if (!e->counted) return fail(e, STBPE_E_STATE, "count the pairs before merging");
    if (e->cfg.world_size > 1) return fail(e, STBPE_E_STATE, "single-rank entry point");
    if (n == 0) return STBPE_OK;
    for (int i = 0; i < 2 * n; ++i)
        if (pairs[i] < 0 || pairs[i] == 0x7FFFFFFF) return fail(e, STBPE_E_ID_OVERFLOW, "Token id overflow: ids must be in [0, 2^31-2]");
    if (first_new_id < 0 || (i64)first_new_id + n - 1 >= 0x7FFFFFFFll)
        return fail(e, STBPE_E_ID_OVERFLOW, "Token id overflow: ids must be in [0, 2^31-2]");
    return run_forced(e, pairs, n, first_new_id, nullptr, (cudaStream_t)stream);
}

STBPE_VISIBLE int stbpe_next_drawn(stbpe_engine *e, int32_t a, int32_t b, int32_t new_id, int32_t most, const uint32_t *draws, int32_t n_draws,
                                   int32_t *n_used, int32_t *n_done, int64_t *count, uint64_t *keys, int64_t cap, int64_t *n_ties, void *stream) {
    if (!e || n_draws < 0 || (n_draws > 0 && (!draws || !n_used)) || !count || !n_ties || !n_done || most < 0 || cap < 0 || (cap > 0 && !keys)) return STBPE_E_BADARG;
    cudaStream_t s = (cudaStream_t)stream;
    CK(cudaSetDevice(e->cfg.device));
    if (!e->counted) return fail(e, STBPE_E_STATE, "count the pairs before selecting");
    if (e->cfg.world_size > 1) return fail(e, STBPE_E_STATE, "single-rank entry point");
    const int given = a >= 0 ? 1 : 0;
    const bool run = given || most > 0;
    *n_done = 0;
    if (n_used) *n_used = 0;
    if (run) {
        if (new_id < 0 || (i64)new_id + most >= 0x7FFFFFFFll || (given && (b < 0 || a == 0x7FFFFFFF || b == 0x7FFFFFFF)))
            return fail(e, STBPE_E_ID_OVERFLOW, "Token id overflow: ids must be in [0, 2^31-2]");
        const int32_t pair[2] = {a, b};
        Draws d = {nullptr, n_draws < STBPE_DRAWS ? n_draws : STBPE_DRAWS, 0};
        if (d.n > 0) {
            if (!e->draws) CK(dev_alloc(e, &e->draws, (size_t)STBPE_DRAWS));
            static_assert(STBPE_DRAWS * sizeof(uint32_t) <= STBPE_PINNED_BYTES - STBPE_PINNED_STATE, "the draws travel through the pinned block");
            void *pin = memcpy((char *)e->pinned.p + STBPE_PINNED_STATE, draws, (size_t)d.n * sizeof(uint32_t));
            CK(cudaMemcpyAsync(e->draws, pin, (size_t)d.n * sizeof(uint32_t), cudaMemcpyHostToDevice, s));
            d.dev = e->draws;
        }
        int rc = run_forced(e, pair, given, new_id, nullptr, s, true, most, n_done, d.n > 0 ? &d : nullptr);
        if (n_used) *n_used = d.used;
        if (rc != STBPE_OK) return rc;
    }
    std::vector<u64> tied;
    i64 c = 0;
    int rc = tied_candidates(e, run, &tied, &c, s);
    if (rc != STBPE_OK) return rc;
    *count = c;
    *n_ties = (i64)tied.size();
    if ((i64)tied.size() <= cap)
        for (size_t i = 0; i < tied.size(); ++i) keys[i] = tied[i];
    return STBPE_OK;
}

STBPE_VISIBLE int stbpe_next_tied(stbpe_engine *e, int32_t a, int32_t b, int32_t new_id, int32_t most, int32_t *n_done, int64_t *count,
                                  uint64_t *keys, int64_t cap, int64_t *n_ties, void *stream) {
    return stbpe_next_drawn(e, a, b, new_id, most, nullptr, 0, nullptr, n_done, count, keys, cap, n_ties, stream);
}

STBPE_VISIBLE int stbpe_token_bytes(const stbpe_engine *e) { return e && e->wide ? 4 : 2; }

static int maybe_repack(stbpe_engine *e, bool force, int *did, cudaStream_t s);

// Keep or drop the pair filter.  A merge whose matches outnumber the tiles visits nearly every tile
// whatever the filter says, while entering its new pairs into the filter costs more than the
// rewrite itself; so the filter is left stale (every merge visits every tile) until the count of the
// last selected pair has fallen to filter_density x tiles, and is then rebuilt from the stream and
// maintained by every later merge.  `h` is the device state as the host has just read it; with
// `layout_changed` the tiles have moved (re-pack), so a filter that is kept must be rebuilt.
static int filter_policy(stbpe_engine *e, const DevState &h, bool layout_changed, cudaStream_t s) {
    if (e->d.n_tiles < 1) return STBPE_OK;
    i64 cnt = h.merges_done > 0 ? h.cur_count : h.peek_count;  // last selected pair, else the best pair of the count
    cnt /= e->cfg.world_size;  // the count is global, the tiles are this rank's
    if (h.merges_done == 0 && h.peek_count == 0) return STBPE_OK;  // nothing has been selected yet
    const bool want = (double)cnt <= e->filter_density * (double)e->d.n_tiles;
    if (want && (!e->filter_valid || layout_changed)) return rebuild_presence(e, s);
    if (layout_changed) {
        clear_skip_state_kernel<<<1, 1, 0, s>>>(e->d, 0);
        CK(cudaGetLastError());
        e->filter_valid = false;
    }
    return STBPE_OK;
}

// Live tokens into the other stream buffer, densely, as 16- or 32-bit tokens; fresh tile records.
static int repack_stream(stbpe_engine *e, bool to_wide, i64 *total, cudaStream_t s) {
    const int nt = e->d.n_tiles;
    i64 *lens = e->rp_lens, *offs = e->rp_offs;
    CK(cudaMemsetAsync(lens + nt, 0, sizeof(i64), s));
    tile_lens_kernel<<<(nt + 255) / 256, 256, 0, s>>>(e->d, lens);
    CK(cudaGetLastError());
    size_t tmp_bytes = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, lens, offs, nt + 1, s);
    if (tmp_bytes > e->rp_tmp_bytes) return fail(e, STBPE_E_STATE, "re-pack scratch too small");
    tmp_bytes = e->rp_tmp_bytes;
    cub::DeviceScan::ExclusiveSum(e->rp_tmp, tmp_bytes, lens, offs, nt + 1, s);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(total, offs + nt, sizeof(i64), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    const size_t want = (size_t)((*total + STBPE_TILE - 1) / STBPE_TILE) * STBPE_TILE * (to_wide ? 4 : 2);
    if (want > e->alt_bytes || !e->tiles_alt) {
        dev_free(e, e->tiles_alt);  // (the stream is idle: it has just been waited for)
        e->tiles_alt = nullptr;
        e->alt_bytes = 0;
        unsigned char *t = nullptr;
        cudaError_t c = dev_alloc(e, &t, want);
        if (c != cudaSuccess) return cuda_fail(e, c, "cudaMalloc second stream buffer");
        e->tiles_alt = t;
        e->alt_bytes = want;
    }
    const int warps = STBPE_REPACK_THREADS / 32;
    const int need = (nt + warps - 1) / warps, grid = need < e->sm_count * 16 ? need : e->sm_count * 16;
    if (e->wide)
        repack_copy_kernel<uint32_t, uint32_t, false><<<grid, STBPE_REPACK_THREADS, 0, s>>>(e->d, offs, (uint32_t *)e->tiles_alt);
    else if (to_wide)
        repack_copy_kernel<uint16_t, uint32_t, false><<<grid, STBPE_REPACK_THREADS, 0, s>>>(e->d, offs, (uint32_t *)e->tiles_alt);
    else
        repack_copy_kernel<uint16_t, uint16_t, false><<<grid, STBPE_REPACK_THREADS, 0, s>>>(e->d, offs, (uint16_t *)e->tiles_alt);
    CK(cudaGetLastError());
    std::swap(e->d.tiles, e->tiles_alt);
    std::swap(e->tiles_bytes, e->alt_bytes);
    e->wide = to_wide;
    e->d.n_tiles = (int)((*total + STBPE_TILE - 1) / STBPE_TILE);
    e->n_tokens = *total;  // capacity in use; the merge log keeps the live counts
    if (e->d.n_tiles > 0) {
        with_tok(e, [&](auto t) {
            init_recs_kernel<decltype(t)><<<(e->d.n_tiles + 255) / 256, 256, 0, s>>>(e->d, *total);
        });
        CK(cudaGetLastError());
    }
    return STBPE_OK;
}

// The 16-bit stream becomes a 32-bit one: an id of 15 bits or more has to go in (a new merge's id, or an id
// of the caller's).  A stream that is still being loaded is converted as it stands, one that merges have
// rewritten is re-packed on the way (its pair filter must then be rebuilt by the caller's policy).
static int widen_stream(stbpe_engine *e, cudaStream_t s) {
    if (e->wide) return STBPE_OK;
    const size_t full = (size_t)e->max_tiles * STBPE_TILE * 4;
    if (e->recs_stale) {
        unsigned char *t = nullptr;
        cudaError_t c = dev_alloc(e, &t, full);
        if (c != cudaSuccess) return cuda_fail(e, c, "cudaMalloc 32-bit token stream");
        if (e->n_tokens > 0) {
            widen_copy_kernel<<<e->sm_count * 8, 256, 0, s>>>((const uint16_t *)e->d.tiles, (uint32_t *)t, e->n_tokens);
            CK(cudaGetLastError());
        }
        CK(cudaStreamSynchronize(s));
        dev_free(e, e->d.tiles);
        dev_free(e, e->tiles_alt);
        e->tiles_alt = nullptr;
        e->alt_bytes = 0;
        e->d.tiles = t;
        e->tiles_bytes = full;
        e->wide = true;
        return STBPE_OK;
    }
    i64 total = 0;
    return repack_stream(e, true, &total, s);
}

// Maintenance between batches of merges: dense re-pack of the stream when at most three quarters of
// the tile capacity in use is live, and the pair-filter policy above.  Synchronises the stream.
// *did (may be NULL) tells whether a re-pack happened.
static int maybe_repack(stbpe_engine *e, bool force, int *did, cudaStream_t s) {
    if (did) *did = 0;
    const int nt = e->d.n_tiles;
    if (nt < 1 || e->recs_stale) return STBPE_OK;
    DevState h;
    if (int rc_ = read_state(e, &h, s)) return rc_;
    if (nt < 2 || (!force && (h.n_live * 4 > (i64)nt * STBPE_TILE * 3 || nt < 64)))  // re-pack at <= 75 % fill
        return filter_policy(e, h, false, s);
    i64 total = 0;
    int rc = repack_stream(e, e->wide, &total, s);
    if (rc != STBPE_OK) return rc;
    rc = filter_policy(e, h, true, s);
    if (rc != STBPE_OK) return rc;
    CK(cudaStreamSynchronize(s));
    e->repacks++;
    e->repacks_since_load++;
    if (did) *did = 1;
    return STBPE_OK;
}

STBPE_VISIBLE int stbpe_repack(stbpe_engine *e, int force, int *did, void *stream) {
    if (!e) return STBPE_E_BADARG;
    CK(cudaSetDevice(e->cfg.device));
    return maybe_repack(e, force != 0, did, (cudaStream_t)stream);
}

__global__ void set_target_kernel(EngineDev e, int target) {
    e.st->target = target;
    e.st->stopped = 0;
    e.st->stop_reason = 0;
    e.st->n_matches = 0;
}

// Runs loop_kernel until a stop rule fires, doing the maintenance it asks for between launches.  `forced`
// (device, n_forced pairs): these merges instead of the best pairs.  *out = the device state at the end.
static int run_loop(stbpe_engine *e, int target, int mode, const int2 *forced, int2 one, int n_forced, int forced_new, DevState *out,
                    cudaStream_t s, bool then_ties = false, int *n_done = nullptr, Draws *draws = nullptr) {
    LoopArgs la;
    int at = 0;
    la.mode = mode;
    la.one = one;
    if (!e->sync_zeroed) {
        CK(cudaMemsetAsync(e->d.sync, 0, 2 * sizeof(LoopSync), s));
        e->sync_zeroed = true;
    }
    if (!e->wide && e->n_tokens >= e->narrow_counts) {  // no count is larger than the stream is long; the largest only falls
        if (int rc_ = choose(e, false, out, s)) return rc_;
        if (out->peek_count >= e->narrow_counts) {
            int rc = widen_stream(e, s);
            if (rc == STBPE_OK) rc = filter_policy(e, *out, true, s);
            if (rc != STBPE_OK) return rc;
        }
    }
    int planes_due = 0;  // a merge that is due needs more planes than this
    int merges = e->merges_done;
    for (;;) {
        const int grid = e->sm_count;  // one CTA per SM; the barrier is no faster with fewer
        la.target = target;
        const int given = at < n_forced ? at : n_forced;
        la.forced = forced ? forced + given : nullptr;
        la.n_forced = n_forced - given;
        la.forced_new = forced_new + at;
        const double fc = e->filter_density * (double)e->d.n_tiles;
        la.filter_count = fc >= 9e18 ? (i64)9000000000000000000ll : (i64)fc;
        la.repack_tiles = 64;
        la.grow_keys = e->table_auto ? (i64)(e->slots / 4) : (i64)0x7FFFFFFFFFFFFFFFll;
        la.ids_below = (int)std::min(ids_below(e), (i64)0x7FFFFFFF);
        la.unit_shift = unit_shift(e, grid);
        la.draws = draws ? draws->dev + draws->used : nullptr;
        la.n_draws = draws ? draws->n - draws->used : 0;
        EngineDev d = e->d;
        // Bits of an id that the loop looks at: as few as all ids allow, old ones and the new ones of the next merges.  For the
        // id that needs more it returns, which costs a launch of 25 to 35 us.  That is earned back where steps are long: over
        // 8192 tiles nine bits lose 22 us against eleven when they serve for 32 merges and gain 14 at 64 (over 2^17 tiles 50 and
        // 123); eleven against fifteen over 16384 tiles -6 at 32 and 29 at 128; thirteen over 65536 tiles -2 at 128 and 38 at
        // 512.  Over 1024 tiles nothing does (eleven for 512 merges: -25), so there they have to serve for all that are left.
        int planes = 15;
        const bool drawing = la.n_draws > 0 && !e->wide;
        if (!e->wide && !drawing) {
            const bool long_steps = e->d.n_tiles >= 8192;
            const i64 next = mode == LOOP_BEST ? (i64)e->cfg.base_vocab + merges : (i64)la.forced_new, left = (i64)target - merges;
            auto enough = [&](int p, i64 worth) {
                const i64 ids = (1 << p) - 1;
                return p > planes_due && la.ids_below < ids && next + (long_steps ? std::min(left, worth) : left) <= ids;
            };
            if (!e->filter_valid && long_steps && enough(9, 64)) planes = 9;
            else if (enough(11, 128)) planes = 11;
            else if (e->filter_valid && enough(13, 512)) planes = 13;
        }
        // Candidates that have run out are collected in front of the launch without waiting for the result: one pass
        // settles the threshold but for tables with very many equal counts, and then the launch comes back at once.
        const bool queued = e->cand_stale;
        if (queued) {
            CK(cudaMemsetAsync(&e->d.st->cand_state, 0, sizeof(int), s));
            if (int rc_ = queue_refill(e, s)) return rc_;
            e->cand_stale = false;
        }
        d.sync = e->d.sync + e->sync_turn;
        la.other_sync = e->d.sync + (e->sync_turn ^= 1);
        void *args[2] = {&d, &la};
        const cudaError_t c = with_tok(e, [&](auto t) {
            typedef decltype(t) T;
            const void *kernel = e->filter_valid ? (const void *)loop_kernel<T, FILTER_ON, 15> : (const void *)loop_kernel<T, FILTER_OFF, 15>;
            if (drawing) kernel = e->filter_valid ? (const void *)loop_kernel<uint16_t, FILTER_ON, 15, true> : (const void *)loop_kernel<uint16_t, FILTER_OFF, 15, true>;
            if (planes == 9) kernel = (const void *)loop_kernel<uint16_t, FILTER_OFF, 9>;
            if (planes == 11) kernel = e->filter_valid ? (const void *)loop_kernel<uint16_t, FILTER_ON, 11> : (const void *)loop_kernel<uint16_t, FILTER_OFF, 11>;
            if (planes == 13) kernel = (const void *)loop_kernel<uint16_t, FILTER_ON, 13>;
            return cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(MergeGeom<T>::THREADS), args,
                                               MergeGeom<T>::BYTES + (STBPE_CAND_CAP + (drawing ? STBPE_DRAWS : 0)) * sizeof(unsigned int), s);
        });
        if (c != cudaSuccess) return cuda_fail(e, c, "cudaLaunchCooperativeKernel");
        if (then_ties) {  // enqueued behind the merge: one round trip for both
            ties_kernel<<<1, 1024, 0, s>>>(e->d);
            CK(cudaGetLastError());
        }
        if (int rc_ = read_state(e, out, s)) return rc_;
        at += out->forced_done;
        merges = out->merges_done;
        if (draws) draws->used += out->draws_used;
        e->made_below = std::max(e->made_below, mode == LOOP_BEST ? (i64)e->cfg.base_vocab + out->merges_done : (i64)forced_new + at);
        if (n_done) *n_done = at;
        int rc = check_error_bits(e, out->error);
        if (rc != STBPE_OK) {
            e->sync_zeroed = false;
            return rc;
        }
        if (out->run_exit == STBPE_EXIT_STOP) return STBPE_OK;
        if (out->run_exit == STBPE_EXIT_GROW) {
            rc = grow_table(e, s);
        } else if (out->run_exit == STBPE_EXIT_REFILL) {
            if (queued && out->forced_done == 0)
                rc = refill_candidates(e, s);
            else
                e->cand_stale = true;
        } else if (out->run_exit == STBPE_EXIT_REPACK) {
            rc = maybe_repack(e, false, nullptr, s);
        } else if (out->run_exit == STBPE_EXIT_FILTER) {
            rc = rebuild_presence(e, s);
        } else if (planes < 15) {
            planes_due = planes;
        } else {
            rc = widen_stream(e, s);
            if (rc == STBPE_OK) rc = filter_policy(e, *out, true, s);
        }
        if (rc != STBPE_OK) return rc;
    }
}

// host-given merges, applied in order as merges of the log
static int run_forced(stbpe_engine *e, const int32_t *pairs, int n, int32_t first_new, int64_t *n_matches, cudaStream_t s,
                      bool then_ties, int most, int *n_done, Draws *draws) {
    DevState h;
    if (!then_ties || !e->merges_known) {
        if (int rc_ = read_state(e, &h, s)) return rc_;
        e->merges_done = h.merges_done;
    }
    if ((i64)e->merges_done + n > e->cfg.max_merges) return fail(e, STBPE_E_CAPACITY, "merge log full");
    if (most > e->cfg.max_merges - e->merges_done - n) most = e->cfg.max_merges - e->merges_done - n;
    if (n > 1 && n > e->forced_cap) {
        dev_free(e, e->forced);
        e->forced = nullptr;
        cudaError_t c = dev_alloc(e, &e->forced, (size_t)n);
        if (c != cudaSuccess) return cuda_fail(e, c, "cudaMalloc merges");
        e->forced_cap = n;
    }
    const void *src = pairs;
    if (n <= 1) {
    } else if ((size_t)n * sizeof(int2) <= STBPE_PINNED_BYTES - STBPE_PINNED_STATE)
        src = memcpy((char *)e->pinned.p + STBPE_PINNED_STATE, pairs, (size_t)n * sizeof(int2));
    if (n > 1) CK(cudaMemcpyAsync(e->forced, src, (size_t)n * sizeof(int2), cudaMemcpyHostToDevice, s));
    if ((i64)first_new + n + most > 65536) e->foreign_ids = true;
    int rc = run_loop(e, e->merges_done + n + most, most > 0 ? LOOP_UNTIED : LOOP_NONE, n > 1 ? e->forced : nullptr,
                      n == 1 ? make_int2(pairs[0], pairs[1]) : make_int2(0, 0), n, first_new, &h, s, then_ties, n_done, draws);
    e->merges_known = rc == STBPE_OK;
    e->merges_done = h.merges_done;
    if (rc == STBPE_OK && n_matches) *n_matches = h.n_matches;
    return rc;
}

STBPE_VISIBLE int stbpe_train(stbpe_engine *e, int32_t n_merges, void *stream) {
    if (!e || n_merges < 0) return STBPE_E_BADARG;
    cudaStream_t s = (cudaStream_t)stream;
    CK(cudaSetDevice(e->cfg.device));
    if (!e->counted) return fail(e, STBPE_E_STATE, "count the pairs before training");
    if (e->cfg.world_size > 1) return fail(e, STBPE_E_STATE, "single-rank entry point");
    DevState h;
    if (!e->merges_known) {
        if (int rc_ = read_state(e, &h, s)) return rc_;
        e->merges_done = h.merges_done;
    }
    i64 target = (i64)e->merges_done + n_merges;
    if (target > e->cfg.max_merges) target = e->cfg.max_merges;
    e->merges_known = false;
    const int rc = run_loop(e, (int)target, LOOP_BEST, nullptr, make_int2(0, 0), 0, 0, &h, s);
    if (rc == STBPE_OK) e->merges_done = h.merges_done, e->merges_known = true;
    return rc;
}

// The merges of stbpe_train one at a time: choose_kernel with the host's look at its result, then merge_kernel, with CUDA
// events around both.
STBPE_VISIBLE int stbpe_train_timed(stbpe_engine *e, int32_t n_merges, float *kernel_ms, void *stream) {
    if (!e || n_merges < 0 || !kernel_ms) return STBPE_E_BADARG;
    cudaStream_t s = (cudaStream_t)stream;
    CK(cudaSetDevice(e->cfg.device));
    if (!e->counted) return fail(e, STBPE_E_STATE, "count the pairs before training");
    if (e->cfg.world_size > 1) return fail(e, STBPE_E_STATE, "single-rank entry point");
    DevState h;
    if (int rc_ = read_state(e, &h, s)) return rc_;
    i64 target = (i64)h.merges_done + n_merges;
    if (target > e->cfg.max_merges) target = e->cfg.max_merges;
    e->made_below = std::max(e->made_below, (i64)e->cfg.base_vocab + target);
    set_target_kernel<<<1, 1, 0, s>>>(e->d, (int)target);
    CK(cudaGetLastError());
    const int todo = (int)(target - h.merges_done);
    e->merges_known = false;
    const int P = 128;
    DevState h2;
    std::vector<cudaEvent_t> ev(3 * P);
    for (auto &x : ev) CK(cudaEventCreate(&x));
    kernel_ms[0] = kernel_ms[1] = kernel_ms[2] = kernel_ms[3] = 0.f;
    int rc = STBPE_OK;
    cudaEvent_t r0, r1;
    CK(cudaEventCreate(&r0));
    CK(cudaEventCreate(&r1));
    for (int base = 0, n = 0; base < todo && rc == STBPE_OK; base += n) {
        {
            int did = 0;
            const bool had_filter = e->filter_valid;
            cudaEventRecord(r0, s);
            rc = maybe_repack(e, false, &did, s);
            cudaEventRecord(r1, s);
            cudaEventSynchronize(r1);
            if (did || had_filter != e->filter_valid) {  // a re-pack and / or a rebuild of the pair filter
                float ms = 0.f;
                cudaEventElapsedTime(&ms, r0, r1);
                kernel_ms[3] += ms;
            }
            if (rc != STBPE_OK) break;
        }
        const int step = (e->filter_valid || e->d.n_tiles < 64) ? P : 32;
        n = todo - base < step ? todo - base : step;
        if (!e->wide && (i64)e->cfg.base_vocab + h.merges_done + base + n >= (i64)Tok<uint16_t>::IDMASK) {
            rc = widen_stream(e, s);
            if (rc == STBPE_OK) {
                CK(cudaMemcpyAsync(&h, e->d.st, sizeof(h), cudaMemcpyDeviceToHost, s));
                CK(cudaStreamSynchronize(s));
                h.merges_done -= base;
                rc = filter_policy(e, h, true, s);
            }
            if (rc != STBPE_OK) break;
        }
        for (int i = 0; i < n && rc == STBPE_OK; ++i) {
            cudaEventRecord(ev[3 * i], s);
            rc = choose(e, true, &h2, s);
            cudaEventRecord(ev[3 * i + 1], s);
            if (rc == STBPE_OK && e->table_auto && (i64)h2.n_keys + 131072 > (i64)(e->slots / 4)) {
                rc = grow_table(e, s);  // every merge adds at most two pairs per id of the vocabulary
                if (rc == STBPE_OK) rc = refill_candidates(e, s);
            }
            if (rc != STBPE_OK) break;
            rc = launch_merge(e, false, s);
            cudaEventRecord(ev[3 * i + 2], s);
        }
        cudaStreamSynchronize(s);
        for (int i = 0; i < n && rc == STBPE_OK; ++i)
            for (int k = 0; k < 2; ++k) {
                float ms = 0.f;
                cudaEventElapsedTime(&ms, ev[3 * i + k], ev[3 * i + k + 1]);
                kernel_ms[k] += ms;
            }
    }
    for (auto &x : ev) cudaEventDestroy(x);
    cudaEventDestroy(r0);
    cudaEventDestroy(r1);
    if (rc != STBPE_OK) return rc;
    rc = choose(e, true, &h2, s);
    return rc != STBPE_OK ? rc : check_device_error(e, s);
}

STBPE_VISIBLE int stbpe_get_state(stbpe_engine *e, stbpe_state *out, void *stream) {
    if (!e || !out) return STBPE_E_BADARG;
    cudaStream_t s = (cudaStream_t)stream;
    CK(cudaSetDevice(e->cfg.device));
    DevState h;
    if (int rc_ = fresh_state(e, s)) return rc_;
    if (int rc_ = read_state(e, &h, s)) return rc_;
    if (e->count_timed && cudaEventElapsedTime(&e->count_ms, e->ev0, e->ev1) == cudaSuccess) e->count_timed = false;
    out->merges_done = h.merges_done;
    out->stop_reason = h.stopped ? h.stop_reason : STBPE_RUNNING;
    out->live_tokens = e->recs_stale ? e->n_tokens : h.n_live;
    out->table_keys = (i64)h.n_keys;
    out->table_slots = (i64)e->slots;
    out->device_error = h.error;
    out->n_tiles = e->d.n_tiles;
    out->fixups = h.n_fixups;
    out->repacks = e->repacks;
    out->work_tiles = h.n_work;
    out->count_kernel_ms = e->count_ms;
    out->count_convert_ms = e->convert_ms;
    out->tile_bytes_in = (i64)h.tile_bytes_in;
    out->tile_bytes_out = (i64)h.tile_bytes_out;
    return STBPE_OK;
}

STBPE_VISIBLE int stbpe_get_merges(stbpe_engine *e, int32_t first, int32_t n, int32_t *merges,
                                   int64_t *counts, int64_t *live_before) {
    if (!e || first < 0 || n < 0 || first + n > e->cfg.max_merges || (n > 0 && !merges))
        return fail(e, STBPE_E_BADARG, "bad merge range");
    CK(cudaSetDevice(e->cfg.device));
    if (n == 0) return STBPE_OK;
    const size_t third = (size_t)n * 8;  // a pair, a count and a number of tokens are eight bytes each
    static_assert(2 * sizeof(int32_t) == 8 && sizeof(i64) == 8, "three columns of eight bytes");
    if (3 * third <= STBPE_PINNED_BYTES - STBPE_PINNED_STATE) {  // one wait for all of them
        char *pin = (char *)e->pinned.p + STBPE_PINNED_STATE;
        CK(cudaMemcpyAsync(pin, e->d.merges + 2 * first, third, cudaMemcpyDeviceToHost, 0));
        if (counts) CK(cudaMemcpyAsync(pin + third, e->d.merge_counts + first, third, cudaMemcpyDeviceToHost, 0));
        if (live_before) CK(cudaMemcpyAsync(pin + 2 * third, e->d.live_before + first, third, cudaMemcpyDeviceToHost, 0));
        CK(cudaStreamSynchronize(0));
        memcpy(merges, pin, third);
        if (counts) memcpy(counts, pin + third, third);
        if (live_before) memcpy(live_before, pin + 2 * third, third);
        return STBPE_OK;
    }
    CK(cudaMemcpy(merges, e->d.merges + 2 * first, third, cudaMemcpyDeviceToHost));
    if (counts) CK(cudaMemcpy(counts, e->d.merge_counts + first, (size_t)n * sizeof(i64), cudaMemcpyDeviceToHost));
    if (live_before) CK(cudaMemcpy(live_before, e->d.live_before + first, (size_t)n * sizeof(i64), cudaMemcpyDeviceToHost));
    return STBPE_OK;
}

STBPE_VISIBLE int stbpe_export_histogram(stbpe_engine *e, uint64_t *keys, int64_t *counts, int64_t cap,
                                         int64_t *n_out, void *stream) {
    if (!e || !n_out || cap < 0) return STBPE_E_BADARG;
    cudaStream_t s = (cudaStream_t)stream;
    CK(cudaSetDevice(e->cfg.device));
    *n_out = 0;
    if (!e->d.table) return STBPE_OK;  // nothing has been counted
    // While every id fits 16 bits and every count 32, the entries are sorted as 32-bit keys with 32-bit counts (half
    // the passes over half the bytes) and widened afterwards.
    if (int rc = fresh_state(e, s)) return rc;
    DevState h;
    if (int rc = read_state(e, &h, s)) return rc;
    const i64 ids = (i64)e->cfg.base_vocab + h.merges_done;
    const bool narrow = e->cfg.world_size == 1 && !e->foreign_ids && e->max_id < 65536 && ids <= 65536 && e->max_tokens < (1ll << 32);
    const size_t elem = narrow ? 4 : 8, side = ((size_t)(cap > 0 ? cap : 1) * elem + 255) & ~(size_t)255;
    size_t tmp_bytes = 0;
    if (narrow)
        cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, (uint32_t *)nullptr, (uint32_t *)nullptr, (uint32_t *)nullptr, (uint32_t *)nullptr, (i64)cap, 0, 32, s);
    else
        cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, (u64 *)nullptr, (u64 *)nullptr, (i64 *)nullptr, (i64 *)nullptr, (i64)cap, 0, 64, s);
    unsigned char *scratch = nullptr;
    CK(dev_alloc(e, &scratch, side * (narrow ? 4 : 2) + tmp_bytes + 256));
    unsigned char *tk = scratch, *tc = scratch + side, *sk = scratch + 2 * side, *sc = scratch + 3 * side, *tmp = scratch + side * (narrow ? 4 : 2);
    CK(cudaMemsetAsync(&e->d.st->export_n, 0, sizeof(i64), s));
    if (narrow)
        export_table_kernel<uint32_t><<<e->sm_count * 4, 512, 0, s>>>(e->d, (uint32_t *)tk, (uint32_t *)tc, cap);
    else
        export_table_kernel<u64><<<e->sm_count * 4, 512, 0, s>>>(e->d, (u64 *)tk, (u64 *)tc, cap);
    CK(cudaGetLastError());
    i64 *n_host = (i64 *)e->pinned.p;
    CK(cudaMemcpyAsync(n_host, &e->d.st->export_n, sizeof(i64), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    const i64 n = *n_host;
    *n_out = n;
    int rc = STBPE_OK;
    if (n > cap) {
        rc = fail(e, STBPE_E_CAPACITY, "pair workspace capacity exceeded");
    } else if (n > 0 && narrow) {
        CK(cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, (uint32_t *)tk, (uint32_t *)sk, (uint32_t *)tc, (uint32_t *)sc, n, 0, 32, s));
        widen_entries_kernel<<<e->sm_count * 8, 256, 0, s>>>((const uint32_t *)sk, (const uint32_t *)sc, n, (u64 *)keys, (i64 *)counts);
    } else if (n > 0) {
        CK(cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, (u64 *)tk, (u64 *)keys, (i64 *)tc, (i64 *)counts, n, 0, 64, s));
    }
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(s));
    dev_free(e, scratch);
    return rc;
}

STBPE_VISIBLE int stbpe_export_ties(stbpe_engine *e, int64_t count, uint64_t *keys, int64_t cap,
                                    int64_t *n_out, void *stream) {
    if (!e || !n_out || cap < 0 || (cap > 0 && !keys)) return STBPE_E_BADARG;
    cudaStream_t s = (cudaStream_t)stream;
    CK(cudaSetDevice(e->cfg.device));
    *n_out = 0;
    if (!e->d.table) return STBPE_OK;  // nothing has been counted
    CK(cudaMemsetAsync(&e->d.st->export_n, 0, sizeof(i64), s));
    export_ties_kernel<<<e->sm_count * 8, 256, 0, s>>>(e->d, count, (u64 *)keys, cap);
    CK(cudaGetLastError());
    i64 n = 0;
    CK(cudaMemcpyAsync(&n, &e->d.st->export_n, sizeof(i64), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    *n_out = n;
    return STBPE_OK;
}

STBPE_VISIBLE int stbpe_export_stream(stbpe_engine *e, int32_t *ids, int64_t cap, int64_t *n_out,
                                      void *stream) {
    if (!e || !n_out) return STBPE_E_BADARG;
    cudaStream_t s = (cudaStream_t)stream;
    CK(cudaSetDevice(e->cfg.device));
    int rc = prepare_stream_state(e, s);
    if (rc != STBPE_OK) return rc;
    const int nt = e->d.n_tiles;
    *n_out = 0;
    if (nt == 0) return STBPE_OK;
    i64 *lens = e->rp_lens, *offs = e->rp_offs, total = 0;
    CK(cudaMemsetAsync(lens + nt, 0, sizeof(i64), s));
    tile_lens_kernel<<<(nt + 255) / 256, 256, 0, s>>>(e->d, lens);
    CK(cudaGetLastError());
    size_t tmp_bytes = e->rp_tmp_bytes;
    cub::DeviceScan::ExclusiveSum(e->rp_tmp, tmp_bytes, lens, offs, nt + 1, s);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(&total, offs + nt, sizeof(i64), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    *n_out = total;
    if (total > cap) return fail(e, STBPE_E_CAPACITY, "export buffer too small");
    const int warps = STBPE_REPACK_THREADS / 32;
    const int need = (nt + warps - 1) / warps, grid = need < e->sm_count * 16 ? need : e->sm_count * 16;
    with_tok(e, [&](auto t) {
        repack_copy_kernel<decltype(t), uint32_t, true><<<grid, STBPE_REPACK_THREADS, 0, s>>>(e->d, offs, (uint32_t *)ids);
    });
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(s));
    return STBPE_OK;
}

// ------------------------------------------------------------------------------- multi-GPU
STBPE_VISIBLE int stbpe_mg_set_buffers(stbpe_engine *e, void *outbox, void *inbox, int64_t cap_per_peer) {
    if (!e || !outbox || !inbox || cap_per_peer < 1) return fail(e, STBPE_E_BADARG, "bad exchange buffers");
    if (e->cfg.world_size < 2) return fail(e, STBPE_E_STATE, "engine was created with world_size 1");
    e->d.outbox = (Slot *)outbox;
    e->d.inbox = (Slot *)inbox;
    e->d.cap_per_peer = cap_per_peer;
    CK(cudaSetDevice(e->cfg.device));
    outbox_reset_kernel<<<1, 64>>>(e->d);
    CK(cudaGetLastError());
    CK(cudaDeviceSynchronize());
    return STBPE_OK;
}

static int launch_drain(stbpe_engine *e, cudaStream_t s) {
    if (!e->d.outbox || e->d.cap_per_peer < 1) return fail(e, STBPE_E_STATE, "call stbpe_mg_set_buffers first");
    drain_ltable_kernel<<<e->sm_count * 2, 256, 0, s>>>(e->d);
    CK(cudaGetLastError());
    return STBPE_OK;
}

STBPE_VISIBLE int stbpe_mg_count_local(stbpe_engine *e, void *stream) {
    if (!e) return STBPE_E_BADARG;
    cudaStream_t s = (cudaStream_t)stream;
    CK(cudaSetDevice(e->cfg.device));
    if (e->cfg.world_size < 2) return fail(e, STBPE_E_STATE, "engine was created with world_size 1");
    int rc = launch_count(e, true, s);
    if (rc != STBPE_OK) return rc;
    rc = launch_drain(e, s);
    if (rc != STBPE_OK) return rc;
    e->counted = true;
    return STBPE_OK;
}

// exchange-only round of the initial histogram: drains what the first round had to keep
STBPE_VISIBLE int stbpe_mg_drain_only(stbpe_engine *e, void *stream) {
    if (!e) return STBPE_E_BADARG;
    cudaStream_t s = (cudaStream_t)stream;
    CK(cudaSetDevice(e->cfg.device));
    if (e->cfg.world_size < 2) return fail(e, STBPE_E_STATE, "engine was created with world_size 1");
    return launch_drain(e, s);
}

STBPE_VISIBLE int stbpe_mg_merge_local(stbpe_engine *e, void *stream) {
    if (!e) return STBPE_E_BADARG;
    cudaStream_t s = (cudaStream_t)stream;
    CK(cudaSetDevice(e->cfg.device));
    if (e->cfg.world_size < 2) return fail(e, STBPE_E_STATE, "engine was created with world_size 1");
    int rc = launch_merge(e, true, s);
    if (rc != STBPE_OK) return rc;
    return launch_drain(e, s);
}

STBPE_VISIBLE int stbpe_mg_apply_inbox(stbpe_engine *e, void *stream) {
    if (!e) return STBPE_E_BADARG;
    cudaStream_t s = (cudaStream_t)stream;
    CK(cudaSetDevice(e->cfg.device));
    if (e->cfg.world_size < 2) return fail(e, STBPE_E_STATE, "engine was created with world_size 1");
    apply_inbox_kernel<<<e->sm_count * 4, 256, 0, s>>>(e->d);
    CK(cudaGetLastError());
    const int all = e->full_refresh_pending ? 1 : 0;
    e->full_refresh_pending = false;
    return launch_refresh(e, all, s);
}

STBPE_VISIBLE int stbpe_mg_candidate(stbpe_engine *e, void *cand_dev, void *stream) {
    if (!e || !cand_dev) return STBPE_E_BADARG;
    cudaStream_t s = (cudaStream_t)stream;
    CK(cudaSetDevice(e->cfg.device));
    select_kernel<<<e->select_grid, STBPE_SELECT_THREADS, 0, s>>>(e->d, 2, e->partial, (i64 *)cand_dev);
    CK(cudaGetLastError());
    return STBPE_OK;
}

STBPE_VISIBLE int stbpe_mg_commit(stbpe_engine *e, const void *all_cands_dev, void *stream) {
    if (!e || !all_cands_dev) return STBPE_E_BADARG;
    cudaStream_t s = (cudaStream_t)stream;
    CK(cudaSetDevice(e->cfg.device));
    commit_kernel<<<1, 1, 0, s>>>(e->d, (const i64 *)all_cands_dev, e->cfg.max_merges);
    CK(cudaGetLastError());
    return STBPE_OK;
}


// ------------------------------------------------------------------ first count of a 16-bit vocabulary, several ranks
// Every rank partitions the pairs of its own rows (first pass); after a barrier that the caller
// provides, the owner of a partition counts it out of every rank's regions over NVLink peer memory
// (second pass).  The next count round (stbpe_mg_count_local, or round 0 of stbpe_mg_peer_run /
// stbpe_mg_run) then finds the table filled and only exchanges, refreshes and selects.
STBPE_VISIBLE int stbpe_mg_wide_export(stbpe_engine *e, void *handle_out64) {
    if (!e || !handle_out64) return STBPE_E_BADARG;
    if (e->cfg.world_size < 2) return fail(e, STBPE_E_STATE, "engine was created with world_size 1");
    if (e->cfg.world_size > STBPE_MAX_PEERS) return fail(e, STBPE_E_BADARG, "at most 16 ranks share buffers");
    if (e->cfg.base_vocab > 65536) return fail(e, STBPE_E_STATE, "the partitioned count needs a vocabulary of at most 65 536 ids");
    CK(cudaSetDevice(e->cfg.device));
    int rc = wide_alloc(e);
    if (rc != STBPE_OK) return rc;
    cudaIpcMemHandle_t h;
    CK(cudaIpcGetMemHandle(&h, e->wide_block));
    memcpy(handle_out64, &h, sizeof(h));
    return STBPE_OK;
}

STBPE_VISIBLE int stbpe_mg_wide_open(stbpe_engine *e, const void *handles, int32_t n_handles) {
    if (!e || !handles) return STBPE_E_BADARG;
    if (!e->wide_block) return fail(e, STBPE_E_STATE, "call stbpe_mg_wide_export first");
    if (n_handles != e->cfg.world_size) return fail(e, STBPE_E_BADARG, "one handle per rank is needed");
    if (e->wide_open) return STBPE_OK;
    CK(cudaSetDevice(e->cfg.device));
    e->wide_peers.world = e->cfg.world_size;
    e->wide_peers.rank = e->cfg.rank;
    for (int r = 0; r < n_handles; ++r) {
        if (r == e->cfg.rank) {
            e->wide_peers.block[r] = e->wide_block;
            continue;
        }
        cudaIpcMemHandle_t h;
        memcpy(&h, (const char *)handles + (size_t)r * sizeof(h), sizeof(h));
        void *p = nullptr;
        CK(cudaIpcOpenMemHandle(&p, h, cudaIpcMemLazyEnablePeerAccess));
        e->wide_mapped[r] = p;
        e->wide_peers.block[r] = (const unsigned char *)p;
    }
    e->wide_open = true;
    return STBPE_OK;
}

// ranks of one process: the allocations are handed over as plain device pointers
STBPE_VISIBLE int stbpe_mg_wide_block(stbpe_engine *e, void **out) {
    if (!e || !out) return STBPE_E_BADARG;
    if (!e->wide_block) return fail(e, STBPE_E_STATE, "call stbpe_mg_wide_export first");
    *out = e->wide_block;
    return STBPE_OK;
}

STBPE_VISIBLE int stbpe_mg_wide_set(stbpe_engine *e, const void *const *blocks, int32_t n) {
    if (!e || !blocks) return STBPE_E_BADARG;
    if (!e->wide_block) return fail(e, STBPE_E_STATE, "call stbpe_mg_wide_export first");
    if (n != e->cfg.world_size) return fail(e, STBPE_E_BADARG, "one block per rank is needed");
    e->wide_peers.world = e->cfg.world_size;
    e->wide_peers.rank = e->cfg.rank;
    for (int r = 0; r < n; ++r) {
        if (r != e->cfg.rank && !blocks[r]) return fail(e, STBPE_E_BADARG, "null block");
        e->wide_peers.block[r] = r == e->cfg.rank ? e->wide_block : (const unsigned char *)blocks[r];
    }
    e->wide_open = true;
    return STBPE_OK;
}

STBPE_VISIBLE int stbpe_mg_wide_pass1(stbpe_engine *e, int32_t *ok, void *stream) {
    if (!e || !ok) return STBPE_E_BADARG;
    cudaStream_t s = (cudaStream_t)stream;
    *ok = 0;
    CK(cudaSetDevice(e->cfg.device));
    if (!e->wide_open) return fail(e, STBPE_E_STATE, "call stbpe_mg_wide_open first");
    const bool fresh = e->recs_stale;
    int rc = count_prologue(e, true, s);
    if (rc != STBPE_OK) return rc;
    if (e->only_bytes || e->d.n_tiles < 1 || !fresh) {
        // nothing to partition here (no rows on this rank, or bytes): an empty first pass, the peers still read it
        CK(cudaMemsetAsync(e->parts.fill, 0, wide_fill_bytes(e->parts.n_cta), s));
        CK(cudaMemsetAsync(e->wide_dense, 0, 65536 * sizeof(u64), s));
        CK(cudaStreamSynchronize(s));
        *ok = e->d.n_tiles < 1 ? 1 : 0;
        return STBPE_OK;
    }
    int good = 0;
    rc = wide_pass1(e, &good, s);
    *ok = good;
    return rc;
}

STBPE_VISIBLE int stbpe_mg_wide_pass2(stbpe_engine *e, void *stream) {
    if (!e) return STBPE_E_BADARG;
    cudaStream_t s = (cudaStream_t)stream;
    CK(cudaSetDevice(e->cfg.device));
    if (!e->wide_open) return fail(e, STBPE_E_STATE, "call stbpe_mg_wide_open first");
    const int world = e->cfg.world_size, n_cta = e->parts.n_cta;
    CK(cudaEventRecord(e->ev0, s));
    dense_peers_to_table_kernel<<<256, 256, 0, s>>>(e->d, e->wide_peers, n_cta);
    CK(cudaGetLastError());
    const int owned = (STBPE_PARTS - e->cfg.rank + world - 1) / world;  // partitions rank, rank + world, ...
    for (int i = 0; i < owned; i += e->part_group) {
        const int n = owned - i < e->part_group ? owned - i : e->part_group;
        partition_table_peers_kernel<<<n_cta * 2 * n, 1024, 0, s>>>(e->d, e->wide_peers, e->cfg.rank + i * world, world, n_cta);
    }
    CK(cudaGetLastError());
    CK(cudaEventRecord(e->ev1, s));
    CK(cudaEventSynchronize(e->ev1));
    CK(cudaEventElapsedTime(&e->convert_ms, e->ev0, e->ev1));
    e->count_ms += e->convert_ms;
    e->wide_counted = true;
    e->full_refresh_pending = true;
    e->counted = true;
    return check_device_error(e, s);
}

// Unmap the peers' buffers (call on every rank, then synchronise the ranks, before any destroys its engine).
STBPE_VISIBLE int stbpe_mg_wide_close(stbpe_engine *e) {
    if (!e) return STBPE_E_BADARG;
    CK(cudaSetDevice(e->cfg.device));
    CK(cudaDeviceSynchronize());
    for (int r = 0; r < STBPE_MAX_PEERS; ++r) {
        if (e->wide_mapped[r]) {
            CK(cudaIpcCloseMemHandle(e->wide_mapped[r]));
            e->wide_mapped[r] = nullptr;
        }
        if (r != e->cfg.rank) e->wide_peers.block[r] = nullptr;
    }
    e->wide_open = false;
    return STBPE_OK;
}

// ------------------------------------------------------------------ rounds over peer memory
// The exchange of a round done by the kernels themselves: every rank owns a mailbox that its peers
// map through CUDA IPC; drain_peer_kernel stores the deltas into the owners' mailboxes,
// select_kernel (mode 3) stores the candidate into every mailbox, and apply_peer_kernel /
// the tail of select_kernel wait (bounded, two seconds) for the senders' flags.  A round is six launches
// and nothing else, so batches of rounds replay as one CUDA graph.  One rank per GPU only.
STBPE_VISIBLE int stbpe_mg_peer_export(stbpe_engine *e, int64_t cap_per_peer, void *handle_out64) {
    if (!e || !handle_out64 || cap_per_peer < 1) return STBPE_E_BADARG;
    if (e->cfg.world_size < 2) return fail(e, STBPE_E_STATE, "engine was created with world_size 1");
    if (e->cfg.world_size > STBPE_MAX_PEERS) return fail(e, STBPE_E_BADARG, "at most 16 ranks share mailboxes");
    if (e->d.cap_per_peer != 0 && e->d.cap_per_peer != cap_per_peer)
        return fail(e, STBPE_E_STATE, "exchange buffers of another capacity are already set");
    CK(cudaSetDevice(e->cfg.device));
    if (!e->mail_own) {
        const size_t bytes = STBPE_MAIL_HEADER_BYTES + (size_t)e->cfg.world_size * (cap_per_peer + 1) * sizeof(Slot);
        cudaError_t c = dev_alloc(e, &e->mail_own, bytes);
        if (c != cudaSuccess) return cuda_fail(e, c, "cudaMalloc mailbox");
        CK(cudaMemset(e->mail_own, 0, bytes));
        CK(cudaDeviceSynchronize());
        e->d.cap_per_peer = cap_per_peer;
    }
    cudaIpcMemHandle_t h;
    CK(cudaIpcGetMemHandle(&h, e->mail_own));
    static_assert(sizeof(h) == 64, "IPC handle size");
    memcpy(handle_out64, &h, sizeof(h));
    return STBPE_OK;
}

STBPE_VISIBLE int stbpe_mg_peer_open(stbpe_engine *e, const void *handles, int32_t n_handles) {
    if (!e || !handles) return STBPE_E_BADARG;
    if (!e->mail_own) return fail(e, STBPE_E_STATE, "call stbpe_mg_peer_export first");
    if (n_handles != e->cfg.world_size) return fail(e, STBPE_E_BADARG, "one handle per rank is needed");
    if (e->peers_open) return STBPE_OK;
    CK(cudaSetDevice(e->cfg.device));
    for (int r = 0; r < n_handles; ++r) {
        if (r == e->cfg.rank) {
            e->d.mail[r] = e->mail_own;
            continue;
        }
        cudaIpcMemHandle_t h;
        memcpy(&h, (const char *)handles + (size_t)r * sizeof(h), sizeof(h));
        void *p = nullptr;
        CK(cudaIpcOpenMemHandle(&p, h, cudaIpcMemLazyEnablePeerAccess));
        e->mail_mapped[r] = p;
        e->d.mail[r] = (unsigned char *)p;
    }
    e->peers_open = true;
    return STBPE_OK;
}

// The same set-up for ranks that live in one process (one GPU each, peer access between the devices
// enabled by the caller): the mailboxes are handed over as plain device pointers.
STBPE_VISIBLE int stbpe_mg_peer_mailbox(stbpe_engine *e, void **out) {
    if (!e || !out) return STBPE_E_BADARG;
    if (!e->mail_own) return fail(e, STBPE_E_STATE, "call stbpe_mg_peer_export first");
    *out = e->mail_own;
    return STBPE_OK;
}

STBPE_VISIBLE int stbpe_mg_peer_set(stbpe_engine *e, const void *const *mailboxes, int32_t n) {
    if (!e || !mailboxes) return STBPE_E_BADARG;
    if (!e->mail_own) return fail(e, STBPE_E_STATE, "call stbpe_mg_peer_export first");
    if (n != e->cfg.world_size) return fail(e, STBPE_E_BADARG, "one mailbox per rank is needed");
    for (int r = 0; r < n; ++r) {
        if (r != e->cfg.rank && !mailboxes[r]) return fail(e, STBPE_E_BADARG, "null mailbox");
        e->d.mail[r] = r == e->cfg.rank ? e->mail_own : (unsigned char *)mailboxes[r];
    }
    e->peers_open = true;
    return STBPE_OK;
}

// Unmap the peers' mailboxes (call on every rank, then synchronise the ranks, before any of them
// destroys its engine).
STBPE_VISIBLE int stbpe_mg_peer_close(stbpe_engine *e) {
    if (!e) return STBPE_E_BADARG;
    CK(cudaSetDevice(e->cfg.device));
    CK(cudaDeviceSynchronize());
    if (e->graph) {
        cudaGraphExecDestroy(e->graph);
        e->graph = nullptr;
    }
    for (int r = 0; r < STBPE_MAX_PEERS; ++r) {
        if (e->mail_mapped[r]) {
            CK(cudaIpcCloseMemHandle(e->mail_mapped[r]));
            e->mail_mapped[r] = nullptr;
        }
        if (r != e->cfg.rank) e->d.mail[r] = nullptr;
    }
    e->peers_open = false;
    return STBPE_OK;
}

static int enqueue_peer_round(stbpe_engine *e, bool count_round, cudaStream_t s) {
    int rc = count_round ? launch_count(e, true, s) : launch_merge(e, true, s);
    if (rc != STBPE_OK) return rc;
    drain_peer_kernel<<<e->sm_count * 2, 256, 0, s>>>(e->d);
    CK(cudaGetLastError());
    apply_peer_kernel<<<e->sm_count * 4, 256, 0, s>>>(e->d);
    CK(cudaGetLastError());
    const int all = e->full_refresh_pending ? 1 : 0;
    e->full_refresh_pending = false;
    rc = launch_refresh(e, all, s);
    if (rc != STBPE_OK) return rc;
    select_kernel<<<e->select_grid, STBPE_SELECT_THREADS, 0, s>>>(e->d, 3, e->partial, e->cand, e->cfg.max_merges);
    CK(cudaGetLastError());
    return STBPE_OK;
}

// first != 0: round 0 counts the local rows.  Enqueues n_rounds rounds; no host synchronisation.
// Every rank must enqueue the same number of rounds.
STBPE_VISIBLE int stbpe_mg_peer_run(stbpe_engine *e, int first, int n_rounds, void *stream) {
    if (!e || n_rounds < 0) return STBPE_E_BADARG;
    if (!e->peers_open) return fail(e, STBPE_E_STATE, "call stbpe_mg_peer_open first");
    cudaStream_t s = (cudaStream_t)stream;
    CK(cudaSetDevice(e->cfg.device));
    int r = 0;
    if (first && n_rounds > 0) {
        int rc = enqueue_peer_round(e, true, s);
        if (rc != STBPE_OK) return rc;
        e->counted = true;
        ++r;
    }
    const int G = 16;  // rounds per graph replay
    while (r < n_rounds) {
        if (e->use_graph && n_rounds - r >= G) {
            if (e->graph && (e->graph_tiles_n != e->d.n_tiles || e->graph_tiles != e->d.tiles || e->graph_wide != e->wide || e->graph_filter != e->d.presence)) {
                cudaGraphExecDestroy(e->graph);
                e->graph = nullptr;
            }
            if (!e->graph) {
                cudaStream_t cs;
                CK(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
                cudaGraph_t g;
                CK(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
                int rc2 = STBPE_OK;
                for (int i = 0; i < G && rc2 == STBPE_OK; ++i) rc2 = enqueue_peer_round(e, false, cs);
                cudaError_t ce = cudaStreamEndCapture(cs, &g);
                if (rc2 != STBPE_OK) {
                    cudaStreamDestroy(cs);
                    return rc2;
                }
                if (ce != cudaSuccess) {
                    cudaStreamDestroy(cs);
                    return cuda_fail(e, ce, "cudaStreamEndCapture");
                }
                ce = cudaGraphInstantiate(&e->graph, g, 0);
                cudaGraphDestroy(g);
                cudaStreamDestroy(cs);
                if (ce != cudaSuccess) return cuda_fail(e, ce, "cudaGraphInstantiate");
                e->graph_tiles_n = e->d.n_tiles;  // the capture froze the stream pointer, n_tiles and the grids
                e->graph_tiles = e->d.tiles;
                e->graph_wide = e->wide;
                e->graph_filter = e->d.presence;
            }
            CK(cudaGraphLaunch(e->graph, s));
            r += G;
        } else {
            int rc = enqueue_peer_round(e, false, s);
            if (rc != STBPE_OK) return rc;
            ++r;
        }
    }
    return STBPE_OK;
}

// ------------------------------------------------------------------ native NCCL round loop
// The rounds of the multi-GPU merge loop issued from C++ on one stream: kernels, an all-to-all of
// the outbox chunks (grouped ncclSend/ncclRecv over NVLink) and an all-gather of the candidates,
// with no Python and no host synchronisation per round.  NCCL is resolved at run time from the
// library that is already loaded in the process (no link-time dependency).
}  // extern "C"

namespace {
struct NcclApi {
    bool ok = false;
    decltype(&ncclGetUniqueId) GetUniqueId = nullptr;
    decltype(&ncclCommInitRank) CommInitRank = nullptr;
    decltype(&ncclCommDestroy) CommDestroy = nullptr;
    decltype(&ncclGroupStart) GroupStart = nullptr;
    decltype(&ncclGroupEnd) GroupEnd = nullptr;
    decltype(&ncclSend) Send = nullptr;
    decltype(&ncclRecv) Recv = nullptr;
    decltype(&ncclAllGather) AllGather = nullptr;
    decltype(&ncclGetErrorString) GetErrorString = nullptr;
};
NcclApi &nccl_api() {
    static NcclApi api;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void *h = dlopen("libnccl.so.2", RTLD_NOW | RTLD_GLOBAL);
        if (!h) h = dlopen("libnccl.so", RTLD_NOW | RTLD_GLOBAL);
        if (h) {
#define NCCL_SYM(field, name) api.field = reinterpret_cast<decltype(api.field)>(dlsym(h, name))
            NCCL_SYM(GetUniqueId, "ncclGetUniqueId");
            NCCL_SYM(CommInitRank, "ncclCommInitRank");
            NCCL_SYM(CommDestroy, "ncclCommDestroy");
            NCCL_SYM(GroupStart, "ncclGroupStart");
            NCCL_SYM(GroupEnd, "ncclGroupEnd");
            NCCL_SYM(Send, "ncclSend");
            NCCL_SYM(Recv, "ncclRecv");
            NCCL_SYM(AllGather, "ncclAllGather");
            NCCL_SYM(GetErrorString, "ncclGetErrorString");
#undef NCCL_SYM
            api.ok = api.GetUniqueId && api.CommInitRank && api.CommDestroy && api.GroupStart && api.GroupEnd &&
                     api.Send && api.Recv && api.AllGather && api.GetErrorString;
        }
    }
    return api;
}
}  // namespace

extern "C" {

#define NCK(call)                                                                              \
    do {                                                                                       \
        ncclResult_t r_ = (call);                                                              \
        if (r_ != ncclSuccess) return fail(e, STBPE_E_CUDA, std::string(#call) + ": " + nccl_api().GetErrorString(r_)); \
    } while (0)

STBPE_VISIBLE int stbpe_mg_nccl_unique_id(void *out128) {
    stbpe_engine *e = nullptr;
    if (!out128) return STBPE_E_BADARG;
    if (!nccl_api().ok) return fail(e, STBPE_E_STATE, "NCCL library not found in this process");
    ncclUniqueId id;
    NCK(nccl_api().GetUniqueId(&id));
    memcpy(out128, &id, sizeof(id));
    return STBPE_OK;
}

STBPE_VISIBLE int stbpe_mg_nccl_init(stbpe_engine *e, const void *id128, int64_t cap_per_peer) {
    if (!e || !id128 || cap_per_peer < 1) return STBPE_E_BADARG;
    if (e->cfg.world_size < 2) return fail(e, STBPE_E_STATE, "engine was created with world_size 1");
    if (!nccl_api().ok) return fail(e, STBPE_E_STATE, "NCCL library not found in this process");
    CK(cudaSetDevice(e->cfg.device));
    if (!e->own_boxes) {
        cudaError_t c;
        const size_t n = (size_t)e->cfg.world_size * (cap_per_peer + 1);
        if ((c = dev_alloc(e, &e->d.outbox, n)) != cudaSuccess) return cuda_fail(e, c, "cudaMalloc outbox");
        if ((c = dev_alloc(e, &e->d.inbox, n)) != cudaSuccess) return cuda_fail(e, c, "cudaMalloc inbox");
        CK(cudaMemset(e->d.outbox, 0, n * sizeof(Slot)));
        CK(cudaMemset(e->d.inbox, 0, n * sizeof(Slot)));
        e->d.cap_per_peer = cap_per_peer;
        e->own_boxes = true;
        outbox_reset_kernel<<<1, 64>>>(e->d);
        CK(cudaGetLastError());
        CK(cudaDeviceSynchronize());
    }
    // one communicator per process and device, shared by every engine created later with the same
    // world size and rank (setting one up costs far more than a training run of a small corpus)
    static ncclComm_t g_comm[64] = {};
    static int g_world[64] = {}, g_rank[64] = {};
    const int dev = e->cfg.device;
    if (dev >= 0 && dev < 64 && g_comm[dev] && g_world[dev] == e->cfg.world_size && g_rank[dev] == e->cfg.rank) {
        e->comm = g_comm[dev];
        return STBPE_OK;
    }
    ncclUniqueId id;
    memcpy(&id, id128, sizeof(id));
    NCK(nccl_api().CommInitRank(&e->comm, e->cfg.world_size, id, e->cfg.rank));
    if (dev >= 0 && dev < 64) {
        g_comm[dev] = e->comm;
        g_world[dev] = e->cfg.world_size;
        g_rank[dev] = e->cfg.rank;
    }
    return STBPE_OK;
}

// first != 0: round 0 counts the local rows; every other round applies the committed merge (or only
// drains, in an exchange-only round).  n_rounds rounds are enqueued on the stream; no synchronisation.
STBPE_VISIBLE int stbpe_mg_run(stbpe_engine *e, int first, int n_rounds, void *stream) {
    if (!e || n_rounds < 0) return STBPE_E_BADARG;
    if (!e->comm) return fail(e, STBPE_E_STATE, "call stbpe_mg_nccl_init first");
    cudaStream_t s = (cudaStream_t)stream;
    CK(cudaSetDevice(e->cfg.device));
    const NcclApi &api = nccl_api();
    const int world = e->cfg.world_size;
    const size_t chunk = (size_t)(e->d.cap_per_peer + 1) * sizeof(Slot);
    for (int r = 0; r < n_rounds; ++r) {
        int rc = (first && r == 0) ? stbpe_mg_count_local(e, stream) : stbpe_mg_merge_local(e, stream);
        if (rc != STBPE_OK) return rc;
        NCK(api.GroupStart());
        for (int p = 0; p < world; ++p) {
            NCK(api.Send((const char *)e->d.outbox + p * chunk, chunk, ncclChar, p, e->comm, s));
            NCK(api.Recv((char *)e->d.inbox + p * chunk, chunk, ncclChar, p, e->comm, s));
        }
        NCK(api.GroupEnd());
        rc = stbpe_mg_apply_inbox(e, stream);
        if (rc != STBPE_OK) return rc;
        rc = stbpe_mg_candidate(e, e->cand, stream);
        if (rc != STBPE_OK) return rc;
        NCK(api.AllGather(e->cand, e->all_cands, 4, ncclInt64, e->comm, s));
        rc = stbpe_mg_commit(e, e->all_cands, stream);
        if (rc != STBPE_OK) return rc;
    }
    return STBPE_OK;
}

}  // extern "C"
