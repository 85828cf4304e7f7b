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

// While it lives, this thread's calls are not seen by a stream capture of another
// library's or thread's (one in the global mode refuses allocations, captures
// and instantiations everywhere, and is invalidated by them).
class OutsideCaptures {
public:
    OutsideCaptures() { cudaThreadExchangeStreamCaptureMode(&mode_); }
    ~OutsideCaptures() { cudaThreadExchangeStreamCaptureMode(&mode_); }
    OutsideCaptures(const OutsideCaptures&) = delete;
    OutsideCaptures& operator=(const OutsideCaptures&) = delete;

private:
    cudaStreamCaptureMode mode_ = cudaStreamCaptureModeRelaxed;
};

// Page-locked, mapped host memory of whole pages: ordinary pages, registered.
// One page takes 0.3 ms and 0.2 to give back, 8 MB of huge pages 0.7 and 0.3;
// cudaHostAlloc takes 2.4 and 0.4 ms for 8 bytes where the process holds no
// other pinned memory, 5.9 and 1.0 for 8 MB.
class PinnedPages {
public:
    PinnedPages() = default;
    PinnedPages(const PinnedPages&) = delete;
    PinnedPages& operator=(const PinnedPages&) = delete;
    ~PinnedPages() { release(); }

    bool allocate(size_t bytes, bool huge);  // false: it cannot be had, nothing is held
    void release();
    void* data() const { return data_; }

private:
    void* base_ = nullptr;
    void* data_ = nullptr;
    size_t mapped_ = 0;
};

// The pinned slots (kThreads * kSlots * kChunk = 8 MB) belong to one engine or
// renderer: allocated by its first read of kAllocFrom bytes or more, given back
// by the destructor.  That read pays for them: 17 / 21 / 31 MB into new arrays
// take 2.7 / 2.9 / 3.1 ms the first time, 1.6 / 1.9 / 2.4 then, one copy 4.2 / 5.1
// / 7.3 (the first time with slots from cudaHostAlloc 7 / 9 / 9 ms).  Reads of
// several threads take turns.
class Readback {
public:
    Readback() = default;
    Readback(const Readback&) = delete;
    Readback& operator=(const Readback&) = delete;
    ~Readback();

    // Copies `bytes` from device memory `src` to host memory `dst` after the
    // work enqueued on `st`; the data is there on return.  Pinned destinations and
    // reads of less than two threads' shares take one cudaMemcpyAsync, and so does
    // every read where the slots cannot be had, or are not there yet and the read
    // would not earn their allocation.
    cudaError_t read(void* dst, const void* src, size_t bytes, cudaStream_t st);

private:
    static constexpr int kThreads = 8;
    static constexpr int kSlots = 2;
    static constexpr size_t kChunk = size_t{512} << 10;
    static constexpr size_t kShare = size_t{4} << 20;  // bytes a thread is worth starting for
    static constexpr size_t kAllocFrom = size_t{16} << 20;

    bool prepare();
    void release();

    std::mutex turn_;
    char* slots_ = nullptr;
    PinnedPages memory_;
    cudaEvent_t done_[kThreads * kSlots] = {};
};

}  // namespace mpm
