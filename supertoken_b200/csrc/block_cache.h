// Device and pinned-host memory that outlives one engine or call.
//
// cudaMalloc / cudaFree cost 0.1-1 ms each for the buffers of an engine (3-9 ms for a whole one, tens of
// milliseconds when other processes of the machine allocate too), the stream-ordered allocator gives its
// memory back at the next synchronisation, and a training run on a small corpus takes a millisecond.  Blocks
// are therefore kept when their owner is done and handed to the next owner that fits.
//
// Bounded: at most `limit` bytes per device (or of pinned host memory) stay cached, the oldest blocks leave
// first; a failing allocation gives everything back and tries again.  Thread-safe.  A block is put back only when
// no work that uses it is pending, so the next owner may use it on any stream.
#pragma once
#include <cuda_runtime.h>

#include <mutex>
#include <vector>

namespace stbpe {

struct Block {
    void *p = nullptr;
    size_t size = 0;
};

class BlockCache {
  public:
    BlockCache(bool pinned, size_t limit) : pinned_(pinned), limit_(limit) {}

    // a block of at least `bytes`; memory of the current device `dev` (pinned blocks: dev = 0)
    cudaError_t get(int dev, size_t bytes, Block *out) {
        const size_t want = rounded(bytes);
        {
            std::lock_guard<std::mutex> lock(mu_);
            std::vector<Block> &f = list(dev);
            int best = -1;
            for (int i = 0; i < (int)f.size(); ++i)
                if (f[i].size >= want && f[i].size <= want + want / 2 && (best < 0 || f[i].size < f[best].size)) best = i;
            if (best >= 0) {
                *out = f[best];
                f.erase(f.begin() + best);
                return cudaSuccess;
            }
        }
        cudaError_t c = raw_alloc(&out->p, want);
        if (c == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            trim(dev, 0);
            c = raw_alloc(&out->p, want);
        }
        out->size = c == cudaSuccess ? want : 0;
        return c;
    }

    void put(int dev, Block b) {
        if (!b.p) return;
        if (b.size > limit_) {
            raw_free(b.p);
            return;
        }
        {
            std::lock_guard<std::mutex> lock(mu_);
            list(dev).push_back(b);
        }
        trim(dev, limit_);
    }

    // give cached blocks back, oldest first, until at most `keep` bytes stay
    void trim(int dev, size_t keep) {
        std::vector<Block> drop;
        {
            std::lock_guard<std::mutex> lock(mu_);
            std::vector<Block> &f = list(dev);
            size_t total = 0;
            for (const Block &b : f) total += b.size;
            while (total > keep) {
                total -= f.front().size;
                drop.push_back(f.front());
                f.erase(f.begin());
            }
        }
        for (const Block &b : drop) raw_free(b.p);
    }

  private:
    // steps of a quarter of a power of two: engines of similar sizes share blocks
    static size_t rounded(size_t n) {
        size_t p = 1 << 16;
        if (n <= p) return p;
        while (p * 2 < n) p *= 2;
        return p + (n - p + p / 4 - 1) / (p / 4) * (p / 4);
    }
    std::vector<Block> &list(int dev) { return free_[dev >= 0 && dev < 64 ? dev : 0]; }
    cudaError_t raw_alloc(void **p, size_t n) { return pinned_ ? cudaMallocHost(p, n) : cudaMalloc(p, n); }
    void raw_free(void *p) {
        if (pinned_)
            cudaFreeHost(p);
        else
            cudaFree(p);
    }
    bool pinned_;
    size_t limit_;
    std::mutex mu_;
    std::vector<Block> free_[64];
};

// never destroyed: at process exit the driver may be gone before static destructors run
inline BlockCache &device_blocks() {
    static BlockCache *c = new BlockCache(false, (size_t)4 << 30);
    return *c;
}
inline BlockCache &pinned_blocks() {
    static BlockCache *c = new BlockCache(true, (size_t)64 << 20);
    return *c;
}

}  // namespace stbpe
