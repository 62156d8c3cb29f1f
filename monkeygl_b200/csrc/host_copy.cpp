// host_copy.cpp -- finished images from pinned staging memory to the caller's
// pageable buffer by several threads.
//
// The bytes come fresh from the device's DMA, so one thread's memcpy runs at
// memory latency (measured 24 us for 512 KB, 47 us for 1 MB, 200 us for 3 MB,
// against 10 / 19 / 55 us for the DMA itself).  Up to three helper threads,
// kept by the process and asleep between images, are woken while the GPU still
// works and then share the copy in 64 KB pieces with the calling thread.  They
// look for it for 200 us and go back to sleep: an image that comes later than
// that is copied by the caller alone.  The caller takes pieces until none is
// left, so a helper that wakes late leaves nothing undone; it waits only for
// pieces that a helper is copying, and gives up its core meanwhile if that takes
// long (the helper may want it).  One caller at a time has the helpers; another
// copies alone, and so does a forked child, which has no helpers and whose
// copies of the locks may be held for good.
#include <string.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <exception>
#include <mutex>
#include <new>
#include <thread>

#include "mk_internal.h"

namespace mk {

namespace {

constexpr size_t kPiece = 64u << 10;
constexpr size_t kHelpMin = 256u << 10;     // smaller images: the caller alone
constexpr int kHelpers = 3;
constexpr auto kSpin = std::chrono::microseconds(200), kWait = std::chrono::microseconds(50);

inline void pause_cpu() {
#if defined(__x86_64__)
    __builtin_ia32_pause();
#else
    std::this_thread::yield();
#endif
}

struct CopyPool {
    const pid_t process = getpid();
    std::mutex owner;                        // held by the caller that has the helpers
    std::mutex mu;
    std::condition_variable cv;
    uint64_t wakes = 0;                      // guarded by mu
    // generation of the copy (high 32 bits) and its pieces not yet taken: a
    // piece is taken by counting one down under the same generation.  Between
    // copies none are left, so a helper that is late for one copy cannot take
    // a piece of the next, whose size it would otherwise see too early.
    std::atomic<uint64_t> ticket{0};
    std::atomic<uint32_t> done{0};
    char *dst = nullptr;                     // written only while no piece is left
    const char *src = nullptr;
    size_t bytes = 0;

    bool take(uint32_t gen) {
        uint64_t t = ticket.load(std::memory_order_acquire);
        for (;;) {
            if ((uint32_t)(t >> 32) != gen || (uint32_t)t == 0) return false;
            if (ticket.compare_exchange_weak(t, t - 1, std::memory_order_acq_rel, std::memory_order_acquire)) break;
        }
        // the piece is this thread's, and the copy cannot end without it
        const uint32_t n = (uint32_t)((bytes + kPiece - 1) / kPiece);
        const size_t off = (size_t)(n - (uint32_t)t) * kPiece;
        memcpy(dst + off, src + off, std::min(kPiece, bytes - off));
        done.fetch_add(1, std::memory_order_release);
        return true;
    }

    void helper() {
        uint64_t seen = 0;
        for (;;) {
            {
                std::unique_lock<std::mutex> lk(mu);
                cv.wait(lk, [&] { return wakes != seen; });
                seen = wakes;
            }
            const auto until = std::chrono::steady_clock::now() + kSpin;
            for (int i = 0;; ++i) {
                const uint64_t t = ticket.load(std::memory_order_acquire);
                if ((uint32_t)t != 0) {
                    while (take((uint32_t)(t >> 32))) {
                    }
                    break;
                }
                if ((i & 63) == 63 && std::chrono::steady_clock::now() > until) break;
                pause_cpu();
            }
        }
    }

    CopyPool() {
        if (std::thread::hardware_concurrency() < 2 * (kHelpers + 1)) return;
        try {
            for (int i = 0; i < kHelpers; ++i) std::thread([this] { helper(); }).detach();
        } catch (const std::exception &) {       // fewer helpers, or none
        }
    }
};

// The process's pool; null in a forked child, and for a caller that comes while
// another makes it.  No lock: one held at a fork would be held in the child.
CopyPool *pool() {
    static std::atomic<CopyPool *> made{nullptr};     // kept until the process exits, like its threads
    static std::atomic<bool> making{false};
    CopyPool *p = made.load(std::memory_order_acquire);
    if (!p) {
        if (making.exchange(true, std::memory_order_acq_rel)) return nullptr;
        p = new (std::nothrow) CopyPool();
        made.store(p, std::memory_order_release);
    }
    return p && p->process == getpid() ? p : nullptr;
}

}  // namespace

void copy_out_soon(size_t bytes) {
    if (bytes < kHelpMin) return;
    CopyPool *p = pool();
    if (!p) return;
    {
        std::lock_guard<std::mutex> lk(p->mu);
        ++p->wakes;
    }
    p->cv.notify_all();
}

void copy_out(void *dst, const void *src, size_t bytes) {
    CopyPool *p = bytes < kHelpMin ? nullptr : pool();
    if (!p || !p->owner.try_lock()) {
        memcpy(dst, src, bytes);
        return;
    }
    const uint32_t n = (uint32_t)((bytes + kPiece - 1) / kPiece);
    const uint32_t gen = (uint32_t)(p->ticket.load(std::memory_order_relaxed) >> 32) + 1;
    p->dst = static_cast<char *>(dst);
    p->src = static_cast<const char *>(src);
    p->bytes = bytes;
    p->done.store(0, std::memory_order_relaxed);
    p->ticket.store((uint64_t)gen << 32 | n, std::memory_order_release);
    while (p->take(gen)) {
    }
    const auto until = std::chrono::steady_clock::now() + kWait;
    bool yield = false;
    for (int i = 1; p->done.load(std::memory_order_acquire) != n; ++i) {
        if (yield) std::this_thread::yield();
        else pause_cpu();
        if (!yield && (i & 63) == 0) yield = std::chrono::steady_clock::now() > until;
    }
    p->owner.unlock();
}

}  // namespace mk
