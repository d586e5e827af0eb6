// host_copy.h - device-to-host copies into pageable memory, through pinned
// pieces and several threads.
//
// A plain cudaMemcpyAsync into pageable memory is staged by the driver on the
// calling thread: about 17 GB/s (9.6 MB: 573 us, 186 us when pinned), plus
// some 15 us a call.  Here the device copies pieces of kPiece bytes into a
// ring of pinned ones at PCIe speed, and the calling thread and up to
// kWorkers helpers copy the pieces that have landed into the caller's memory
// (also spreading the page faults of memory not touched before).  Measured
// with 16 cores: 9.6 MB of Stars 638 -> 340 us, a host step of 300,000
// particles into pageable memory 1,529 -> 651 us (its 64 plain chunk copies
// cost more than its walk), a 1920 x 1080 frame 799 -> 557 us.  Two, four and
// eight threads copy 9.6 MB in 358, 264 and 423 us.  The helpers are
// called when a piece is queued and when one has landed, and sleep behind queued
// steps and between the chunks of a long walk (CPU time of a host step of
// 1,000,000 particles at theta 0.5, 3.06 ms: 8.6 ms with helpers awake from the
// first chunk to the last, 6.6 so; called by landed pieces alone, 5.2, but a host
// step of 300,000 took 0.65 ms in place of 0.60).
//
// One ring and its threads serve the process, kept while a context that copies
// lives and given back with the last.  Making them takes 4 to 5 ms, which a
// program with few copies does not get back (its first copy of 1 MiB took 5.1 ms
// in place of 0.19, of 9.6 MB 5.0 in place of 0.8): copies go plainly until
// kEarned bytes have, which has cost as much.  A copy takes the ring for itself
// (begin() fails while another thread has it, and callers then copy plainly).
#pragma once
#include <cstddef>
#include <cuda_runtime.h>

namespace gcs {

class HostCopy {
  public:
    static constexpr size_t kPiece = 512 << 10;
    static constexpr int kSlots = 8;
    static constexpr int kWorkers = 3;
    static constexpr size_t kWorth = 1 << 20;  // smaller copies go plainly
    static constexpr size_t kEarned = 64 << 20;

    // The process's instance, counted by user; nullptr where there is no second
    // core.
    static HostCopy* acquire();
    static void release();

    bool begin(size_t bytes);  // take it for a copy of bytes; false: copy plainly
    // Queue a copy of `bytes` from device memory on `st`; blocks (working on
    // landed pieces) while the ring is full.  Nothing is queued after an error.
    void add(void* dst, const void* src, size_t bytes, cudaStream_t st);
    void work();            // copy one landed piece, if there is one
    cudaError_t finish();   // wait for everything queued, and give it back

  private:
    struct Impl;
    Impl* impl = nullptr;
    HostCopy() = default;
    ~HostCopy();
    void poll();
};

// Whether p is ordinary pageable host memory (false: pinned, managed or
// device memory, which cudaMemcpyAsync copies to directly).
bool is_pageable(const void* p);

}  // namespace gcs
