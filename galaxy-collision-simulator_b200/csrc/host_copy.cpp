// host_copy.cpp - see host_copy.h.
#include "host_copy.h"

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

#include <csignal>
#include <unistd.h>

namespace gcs {

namespace {

inline void relax() {
#if defined(__x86_64__)
    __builtin_ia32_pause();
#endif
}

std::mutex g_mu;
HostCopy* g_copy = nullptr;
int g_users = 0;

}  // namespace

struct HostCopy::Impl {
    struct Piece {
        char* dst;
        size_t bytes;
    };
    char* ring = nullptr;                 // pinned, kSlots pieces
    cudaEvent_t landed_ev[kSlots] = {};   // of the device current at begin()
    int device = -1;
    Piece piece[kSlots];
    // piece numbers, never reset
    std::atomic<uint64_t> landed{0};      // pieces whose device copy is done
    std::atomic<uint64_t> claimed{0};     // pieces taken by a copying thread
    std::atomic<uint64_t> done[kSlots];   // piece number + 1 last copied out of the slot
    uint64_t queued = 0;                  // owner's
    cudaError_t error = cudaSuccess;      // owner's
    std::mutex own;                       // the running copy
    std::mutex mu;                        // wakes the helpers
    std::condition_variable cv;
    std::atomic<int> asleep{0};           // helpers that wait for a call
    std::atomic<uint64_t> calls{0};
    bool stop = false;
    size_t plain = 0;                     // bytes copied plainly so far (owner's)
    bool tried = false;                   // set_up has been called
    pid_t owner = 0;                      // the process that has the helpers
    std::vector<std::thread> threads;

    // The ring and the helpers; false: there is no pinned memory.
    bool set_up() {
        if (tried) return ring != nullptr;
        tried = true;
        owner = getpid();
        for (auto& d : done) d.store(0, std::memory_order_relaxed);
        if (cudaHostAlloc(reinterpret_cast<void**>(&ring), kPiece * kSlots, cudaHostAllocPortable) != cudaSuccess) {
            cudaGetLastError();
            ring = nullptr;
            return false;
        }
        // the process's signals stay with its own threads: helpers inherit this
        // mask and take none
        sigset_t every, before;
        sigfillset(&every);
        const bool masked = pthread_sigmask(SIG_SETMASK, &every, &before) == 0;
        try {
            const int cores = (int)std::thread::hardware_concurrency();
            for (int k = 0; k < std::min(kWorkers, cores - 1); ++k) threads.emplace_back([this] { help(); });
        } catch (...) {  // fewer threads, or none: the caller's own still copies
        }
        if (masked) pthread_sigmask(SIG_SETMASK, &before, nullptr);
        return true;
    }

    bool copy_one() {
        uint64_t i = claimed.load(std::memory_order_relaxed);
        if (i >= landed.load(std::memory_order_acquire)) return false;
        if (!claimed.compare_exchange_strong(i, i + 1, std::memory_order_relaxed)) return false;
        const int s = (int)(i % kSlots);
        std::memcpy(piece[s].dst, ring + (size_t)s * kPiece, piece[s].bytes);
        done[s].store(i + 1, std::memory_order_release);
        return true;
    }
    // A helper sleeps until it is called: when a piece is queued, so that it
    // wakes while the piece travels, and when one has landed (its copy may have
    // been queued behind a long step).  It goes back to sleep when no piece has
    // landed for kFirst after a call or kAwake after its last one: the chunks of
    // a host step can be far apart while the device walks.  (asleep and calls
    // are sequentially consistent: either the helper sees the call or wake()
    // sees the helper.)
    void help() {
        using Clock = std::chrono::steady_clock;
        for (uint64_t seen = 0;;) {
            {
                std::unique_lock<std::mutex> lk(mu);
                ++asleep;
                cv.wait(lk, [&] { return stop || calls.load() != seen; });
                --asleep;
                if (stop) return;
            }
            for (Clock::time_point until = Clock::now() + kFirst; Clock::now() < until;) {
                if (copy_one()) until = Clock::now() + kAwake;
                else for (int k = 0; k < 4; ++k) relax();
                seen = calls.load();  // calls while awake need no other turn
            }
        }
    }
    void wake() {
        ++calls;
        if (asleep.load() == 0) return;
        { std::lock_guard<std::mutex> lk(mu); }
        cv.notify_all();
    }
    static constexpr std::chrono::microseconds kFirst{50}, kAwake{15};
    void drop_events() {
        for (cudaEvent_t& e : landed_ev) {
            if (e) cudaEventDestroy(e);
            e = nullptr;
        }
        device = -1;
    }
    ~Impl() {
        {
            std::lock_guard<std::mutex> lk(mu);
            stop = true;
        }
        cv.notify_all();
        for (std::thread& t : threads) t.join();
        drop_events();
        if (ring) cudaFreeHost(ring);
    }
};

HostCopy::~HostCopy() { delete impl; }

HostCopy* HostCopy::acquire() {
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_copy) {
        if (std::thread::hardware_concurrency() < 2) return nullptr;
        Impl* im = new (std::nothrow) Impl();
        if (!im) return nullptr;
        g_copy = new (std::nothrow) HostCopy();
        if (!g_copy) {
            delete im;
            return nullptr;
        }
        g_copy->impl = im;
    }
    ++g_users;
    return g_copy;
}

void HostCopy::release() {
    HostCopy* last = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if (--g_users == 0) {
            last = g_copy;
            g_copy = nullptr;
        }
    }
    // a forked child has the object but not its threads: joining them would
    // wait for good, so there it is left to the end of the process
    if (last && (!last->impl->tried || last->impl->owner == getpid())) delete last;
}

bool HostCopy::begin(size_t bytes) {
    Impl& m = *impl;
    if (!m.own.try_lock()) return false;
    if (m.plain < kEarned) {
        m.plain += std::min(bytes, kEarned);
        m.own.unlock();
        return false;
    }
    if (!m.set_up()) {
        m.own.unlock();
        return false;
    }
    int dev = -1;
    bool ok = cudaGetDevice(&dev) == cudaSuccess;
    if (ok && dev != m.device) {  // events belong to a device
        m.drop_events();
        for (cudaEvent_t& e : m.landed_ev)
            ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
        if (ok) m.device = dev;
        else m.drop_events();
    }
    if (!ok) {
        cudaGetLastError();
        m.own.unlock();
        return false;
    }
    // the counters go on from the last copy (a helper may still be looking at
    // them); pieces that an error kept from landing are numbered again
    m.queued = m.landed.load(std::memory_order_relaxed);
    m.error = cudaSuccess;
    return true;
}

// Take note of pieces that have landed (in order).
void HostCopy::poll() {
    Impl& m = *impl;
    const uint64_t before = m.landed.load(std::memory_order_relaxed);
    uint64_t i = before;
    while (i < m.queued && m.error == cudaSuccess) {
        const cudaError_t e = cudaEventQuery(m.landed_ev[i % kSlots]);
        if (e == cudaErrorNotReady) break;
        if (e != cudaSuccess) {
            m.error = e;
            break;
        }
        m.landed.store(++i, std::memory_order_release);
    }
    if (i > before) m.wake();
}

void HostCopy::work() {
    poll();
    if (!impl->copy_one()) relax();
}

void HostCopy::add(void* dst, const void* src, size_t bytes, cudaStream_t st) {
    Impl& m = *impl;
    for (size_t at = 0; at < bytes && m.error == cudaSuccess; at += kPiece) {
        const uint64_t i = m.queued;
        const int s = (int)(i % kSlots);
        // the slot's last piece has been copied out
        while (i >= kSlots && m.done[s].load(std::memory_order_acquire) != i - kSlots + 1 && m.error == cudaSuccess)
            work();
        if (m.error != cudaSuccess) return;
        m.piece[s].dst = static_cast<char*>(dst) + at;
        m.piece[s].bytes = std::min(kPiece, bytes - at);
        cudaError_t e = cudaMemcpyAsync(m.ring + (size_t)s * kPiece, static_cast<const char*>(src) + at,
                                        m.piece[s].bytes, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaEventRecord(m.landed_ev[s], st);
        if (e != cudaSuccess) {
            m.error = e;
            return;
        }
        m.queued = i + 1;
        m.wake();
        poll();
    }
}

cudaError_t HostCopy::finish() {
    Impl& m = *impl;
    const auto copied = [&] {
        const uint64_t n = m.landed.load(std::memory_order_relaxed);
        // every landed piece: the last kSlots of them say so themselves, the
        // ones before made room for them
        for (uint64_t i = n > kSlots ? n - kSlots : 0; i < n; ++i)
            if (m.done[i % kSlots].load(std::memory_order_acquire) != i + 1) return false;
        return true;
    };
    while (m.error == cudaSuccess && m.landed.load(std::memory_order_relaxed) < m.queued) work();
    while (!copied()) work();
    // after an error no device copy may still be on its way into the ring
    if (m.error != cudaSuccess)
        for (int s = 0; s < kSlots; ++s)
            if (m.landed_ev[s]) cudaEventSynchronize(m.landed_ev[s]);
    const cudaError_t e = m.error;
    m.own.unlock();
    return e;
}

bool is_pageable(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

}  // namespace gcs
