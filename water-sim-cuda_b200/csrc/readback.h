// Read-back of large results into pageable host memory.
//
// cudaMemcpy to pageable memory copies through the driver's staging buffer on
// one host thread, and into a fresh allocation (what numpy hands out for every
// large array) that thread also takes each page's first fault: 5 GB/s there,
// 20 GB/s into touched pages, where the link carries 57.  Here up to kThreads
// threads share the destination out in contiguous ranges; each copies its own
// in chunks through two pinned slots, so the link, the faults and the copies of
// all threads overlap.  A 1920 x 1600 image (46 MB, into new arrays) rendered and
// read: 9.8 / 3.2 ms on 16 cores (4 threads 3.9, 16 threads 3.0; 2 MB a thread
// 2.9, but then 8.4 MB into touched pages takes 12 % longer than in one copy
// instead of as long).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <mutex>

namespace mpm {

// The pinned slots (kThreads * kSlots * kChunk = 8 MB) belong to one engine or
// renderer and are given back by its destructor.  Having them costs 4 to 8 ms
// once, what 25 to 50 MB of reads into fresh pages gain, so they are allocated
// when the object's reads of kCountFrom bytes or more have come to kAllocFrom:
// allocated by the first such read, one of 17 / 21 / 31 MB took 6.9 / 12 / 10 ms,
// plain ones 4.4 / 5.4 / 7.3; a first read of 208 MB takes 18 ms with them and 45
// without.  Reads of several threads take turns.
class Readback {
public:
    Readback() = default;
    Readback(const Readback&) = delete;
    Readback& operator=(const Readback&) = delete;
    ~Readback();

    // Copies `bytes` from device memory `src` to host memory `dst` after the
    // work enqueued on `st`; the data is there on return.  Pinned destinations and
    // reads of less than two threads' shares take one cudaMemcpyAsync, and so does
    // every read where the slots cannot be had, or are not there yet and the
    // reads so far would not earn their allocation.
    cudaError_t read(void* dst, const void* src, size_t bytes, cudaStream_t st);

private:
    static constexpr int kThreads = 8;
    static constexpr int kSlots = 2;
    static constexpr size_t kChunk = size_t{512} << 10;
    static constexpr size_t kShare = size_t{4} << 20;  // bytes a thread is worth starting for
    static constexpr size_t kCountFrom = size_t{16} << 20;
    static constexpr size_t kAllocFrom = size_t{128} << 20;

    bool prepare();
    void release();

    std::mutex turn_;
    size_t read_ = 0;  // bytes of the reads counted before the slots were there
    char* slots_ = nullptr;
    cudaEvent_t done_[kThreads * kSlots] = {};
};

}  // namespace mpm
