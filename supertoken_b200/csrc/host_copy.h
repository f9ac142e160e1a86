// Host memory -> device staging buffer.
//
// A copy from pageable memory runs at about 9 GB/s, because the driver stages it with one thread and the caller
// waits.  Here the bytes go through a ring of pinned chunks that a few threads fill while the copy engine
// drains the chunks before: 64 MB of pageable bytes in 2.6 ms instead of 6.5.  Pinned sources skip the ring.
#pragma once
#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <thread>

#include "block_cache.h"

namespace stbpe {

// memcpy by several threads; one copy at a time (the caller's thread takes part)
class CopyPool {
  public:
    static CopyPool &instance() {
        static CopyPool *p = new CopyPool();  // never destroyed: its threads wait until the process ends
        return *p;
    }
    void copy(void *dst, const void *src, size_t n) {
        std::lock_guard<std::mutex> one(call_mu_);
        const int parts = (int)threads_.size() + 1;
        {
            std::lock_guard<std::mutex> lock(mu_);
            dst_ = (char *)dst, src_ = (const char *)src, n_ = n;
            left_ = parts - 1;
            ++round_;
        }
        wake_.notify_all();
        slice(parts - 1, parts);
        std::unique_lock<std::mutex> lock(mu_);
        done_.wait(lock, [&] { return left_ == 0; });
    }

  private:
    CopyPool() {
        const int n = std::max(1, std::min(4, (int)std::thread::hardware_concurrency() / 2));
        for (int i = 0; i + 1 < n; ++i) {
            threads_.emplace_back([this, i, n] {
                for (unsigned long long seen = 0;;) {
                    {
                        std::unique_lock<std::mutex> lock(mu_);
                        wake_.wait(lock, [&] { return round_ != seen; });
                        seen = round_;
                    }
                    slice(i, n);
                    std::lock_guard<std::mutex> lock(mu_);
                    if (--left_ == 0) done_.notify_one();
                }
            });
            threads_.back().detach();
        }
    }
    void slice(int i, int parts) {
        const size_t step = (n_ / parts + 63) & ~(size_t)63, lo = std::min(n_, step * i), hi = i + 1 == parts ? n_ : std::min(n_, step * (i + 1));
        if (hi > lo) memcpy(dst_ + lo, src_ + lo, hi - lo);
    }
    std::mutex call_mu_, mu_;
    std::condition_variable wake_, done_;
    std::vector<std::thread> threads_;
    char *dst_ = nullptr;
    const char *src_ = nullptr;
    size_t n_ = 0;
    int left_ = 0;
    unsigned long long round_ = 0;
};

// Pieces of a host buffer on their way through a staging buffer of two halves: piece k + 2 overwrites the half of
// piece k once its consumer has read it.  consume(device pointer, element offset, elements) enqueues work on
// `s`; the call returns when all copies have left the host buffer.
template <typename F>
cudaError_t staged_copy(const void *host, size_t n, size_t elem, bool pageable, void *stage, size_t half_bytes, cudaStream_t s, F &&consume) {
    constexpr size_t CHUNK = (size_t)8 << 20;
    constexpr int RING = 3;
    cudaStream_t cs = nullptr;
    cudaEvent_t landed = nullptr, eaten[2] = {nullptr, nullptr}, left[RING] = {};
    Block ring;
    cudaError_t c = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
    auto event = [&](cudaEvent_t *ev) {
        if (c == cudaSuccess) c = cudaEventCreateWithFlags(ev, cudaEventDisableTiming);
    };
    event(&landed);
    for (auto &ev : eaten) event(&ev);
    if (c == cudaSuccess && pageable) c = pinned_blocks().get(0, CHUNK * RING, &ring);
    if (pageable)
        for (auto &ev : left) event(&ev);
    if (c == cudaSuccess) c = cudaEventRecord(landed, s);  // the staging buffer is free once s got here
    if (c == cudaSuccess) c = cudaStreamWaitEvent(cs, landed, 0);
    const size_t piece = half_bytes / elem;
    int slot = 0, used = 0;
    for (size_t at = 0, k = 0; at < n && c == cudaSuccess; at += piece, ++k) {
        const size_t cnt = std::min(piece, n - at), bytes = cnt * elem;
        char *dst = (char *)stage + (k & 1) * half_bytes;
        const char *src = (const char *)host + at * elem;
        if (k >= 2) c = cudaStreamWaitEvent(cs, eaten[k & 1], 0);
        if (!pageable) {
            if (c == cudaSuccess) c = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, cs);
        } else {
            for (size_t o = 0; o < bytes && c == cudaSuccess; o += CHUNK) {
                const size_t m = std::min(CHUNK, bytes - o);
                char *pin = (char *)ring.p + (size_t)slot * CHUNK;
                if (used >= RING) c = cudaEventSynchronize(left[slot]);
                if (c != cudaSuccess) break;
                CopyPool::instance().copy(pin, src + o, m);
                c = cudaMemcpyAsync(dst + o, pin, m, cudaMemcpyHostToDevice, cs);
                if (c == cudaSuccess) c = cudaEventRecord(left[slot], cs);
                slot = (slot + 1) % RING;
                ++used;
            }
        }
        if (c == cudaSuccess) c = cudaEventRecord(landed, cs);
        if (c == cudaSuccess) c = cudaStreamWaitEvent(s, landed, 0);  // waits for the record just made
        if (c == cudaSuccess) c = consume(dst, at, cnt);
        if (c == cudaSuccess) c = cudaEventRecord(eaten[k & 1], s);
    }
    if (cs) {
        const cudaError_t d = cudaStreamSynchronize(cs);
        if (c == cudaSuccess) c = d;
    }
    pinned_blocks().put(0, ring);
    if (landed) cudaEventDestroy(landed);
    for (auto &ev : eaten)
        if (ev) cudaEventDestroy(ev);
    for (auto &ev : left)
        if (ev) cudaEventDestroy(ev);
    if (cs) cudaStreamDestroy(cs);
    return c;
}

}  // namespace stbpe
