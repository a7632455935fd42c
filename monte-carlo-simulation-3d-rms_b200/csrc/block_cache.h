// block_cache.h -- memory of finished work, kept for the next.
//
// A program that makes a simulation per call (a fit through torch makes two per
// iteration) spent 10 to 40 ms of each in cudaMalloc, cudaMallocHost and their
// frees: a pass of waveform gradients over 1e5 walkers took 48 to 70 ms, 34.5
// with the cache.  The contraction's workspaces come from it too.
//  - bounded: at most `most` bytes, and a block that 256 requests in a row have
//    passed over is freed; all blocks are freed when an allocation fails and when
//    a program asks (rms_memory_trim);
//  - blocks go to a request they are at most a quarter (and 1 MB) larger than, on
//    their own device;
//  - one mutex; a block enters only when no work on it is in flight (every call
//    waits for its stream before it returns, on its error paths too: StreamWait in
//    rms_api.cpp), so the next owner may use any stream.  Nothing here waits for
//    the device: that would wait for other threads' simulations, and would break a
//    capture that another thread has begun.
#ifndef RMS_BLOCK_CACHE_H
#define RMS_BLOCK_CACHE_H

#include <cstddef>
#include <mutex>
#include <new>
#include <vector>

namespace rms {

class BlockCache {
  public:
    // alloc: a block of n bytes on the calling thread's device, 0 or an error
    // code (and then *p is not looked at); release: gives one back, whatever the
    // calling thread's device
    using Alloc = int (*)(void** p, size_t n);
    using Release = void (*)(void* p);
    BlockCache(Alloc alloc, Release release, size_t most) : alloc_(alloc), release_(release), most_(most) {}

    // A block of at least `bytes` on `device`, the calling thread's: 0, or the
    // allocation's error code, *p null.
    int take(size_t bytes, int device, void** p, size_t* got) {
        std::lock_guard<std::mutex> lk(mu_);
        ++now_;
        int best = -1;
        for (int k = 0; k < (int)free_.size(); ++k) {
            const Block& b = free_[k];
            if (b.device == device && b.n >= bytes && b.n <= bytes + bytes / 4 + ((size_t)1 << 20) &&
                (best < 0 || b.n < free_[best].n))
                best = k;
        }
        if (best >= 0) {
            *p = free_[best].p;
            *got = free_[best].n;
            held_ -= free_[best].n;
            free_.erase(free_.begin() + best);
        }
        drop_passed_over();
        if (best >= 0) return 0;
        int e = alloc_(p, bytes);
        if (e && !free_.empty()) {
            drop([](const Block&) { return true; });
            e = alloc_(p, bytes);
        }
        if (e) *p = nullptr;
        *got = bytes;
        return e;
    }

    // Takes a block back; no work on it is in flight.
    void give(void* p, size_t n, int device) {
        if (n > most_) {
            release_(p);
            return;
        }
        std::lock_guard<std::mutex> lk(mu_);
        try {
            free_.push_back(Block{p, n, device, now_});
        } catch (const std::bad_alloc&) {   // (called from destructors and C entries)
            release_(p);
            return;
        }
        held_ += n;
        drop_passed_over();
        while (held_ > most_) {   // the oldest first
            const long oldest = free_.front().since;
            bool one = false;
            drop([&](const Block& b) { return !one && b.since == oldest && (one = true); });
        }
    }

    // Frees every block; returns their bytes.
    size_t trim() {
        std::lock_guard<std::mutex> lk(mu_);
        const size_t n = held_;
        drop([](const Block&) { return true; });
        return n;
    }

    // Bytes of blocks on `device`: free memory to who asks for it here.
    size_t held(int device) {
        std::lock_guard<std::mutex> lk(mu_);
        size_t n = 0;
        for (const Block& b : free_)
            if (b.device == device) n += b.n;
        return n;
    }

  private:
    struct Block {
        void* p;
        size_t n;
        int device;
        long since;
    };
    void drop_passed_over() {
        drop([this](const Block& b) { return now_ - b.since > 256; });
    }
    template <class F>
    void drop(F which) {
        for (size_t k = 0; k < free_.size();) {
            if (which(free_[k])) {
                release_(free_[k].p);
                held_ -= free_[k].n;
                free_.erase(free_.begin() + k);
            } else {
                ++k;
            }
        }
    }
    const Alloc alloc_;
    const Release release_;
    const size_t most_;
    std::mutex mu_;
    std::vector<Block> free_;   // oldest first
    size_t held_ = 0;
    long now_ = 0;
};

// The library's caches (rms_api.cpp): device memory (at most 4 GiB) and pinned
// host memory (256 MiB).
BlockCache& block_cache(bool host);

}  // namespace rms
#endif
