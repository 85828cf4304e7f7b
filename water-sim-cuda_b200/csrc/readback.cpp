#include "readback.h"

#include <sys/mman.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <thread>

namespace mpm {

Readback::~Readback() { release(); }

void Readback::release() {
    for (cudaEvent_t& e : done_) {
        if (e) cudaEventDestroy(e);
        e = nullptr;
    }
    slots_ = nullptr;
    memory_.release();
}

bool PinnedPages::allocate(size_t bytes, bool huge) {
    constexpr size_t kHugePage = size_t{2} << 20;
    const size_t align = huge ? kHugePage : 1;
    mapped_ = bytes + align - 1;
    base_ = mmap(nullptr, mapped_, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (base_ == MAP_FAILED) {
        base_ = nullptr;
        return false;
    }
    const uintptr_t at = (reinterpret_cast<uintptr_t>(base_) + align - 1) / align * align;
    data_ = reinterpret_cast<void*>(at);
    if (huge) madvise(data_, bytes, MADV_HUGEPAGE);  // only a hint
    // A forked child must not share the pages: the first write after a fork
    // could otherwise leave this process with a copy the device knows nothing of.
    madvise(data_, bytes, MADV_DONTFORK);
    if (cudaHostRegister(data_, bytes, cudaHostRegisterMapped) == cudaSuccess) return true;
    cudaGetLastError();
    munmap(base_, mapped_);
    base_ = data_ = nullptr;
    return false;
}

void PinnedPages::release() {
    if (!base_) return;
    cudaHostUnregister(data_);
    munmap(base_, mapped_);
    base_ = data_ = nullptr;
}

bool Readback::prepare() {
    if (slots_) return true;
    const OutsideCaptures outside;
    cudaError_t err = memory_.allocate(kThreads * kSlots * kChunk, true) ? cudaSuccess : cudaErrorMemoryAllocation;
    slots_ = static_cast<char*>(memory_.data());
    for (int k = 0; k < kThreads * kSlots && err == cudaSuccess; ++k)
        err = cudaEventCreateWithFlags(&done_[k], cudaEventDisableTiming);
    if (err == cudaSuccess) return true;
    cudaGetLastError();
    release();
    return false;
}

cudaError_t Readback::read(void* dst, const void* src, size_t bytes, cudaStream_t st) {
    const auto plain = [&] {
        const cudaError_t err = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
        return err == cudaSuccess ? cudaStreamSynchronize(st) : err;
    };
    const int threads = static_cast<int>(
        std::min({static_cast<size_t>(kThreads), static_cast<size_t>(std::thread::hardware_concurrency()), bytes / kShare}));
    if (threads < 2) return plain();
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, dst) != cudaSuccess) {
        cudaGetLastError();
        return plain();
    }
    if (at.type != cudaMemoryTypeUnregistered) return plain();
    std::lock_guard<std::mutex> turn(turn_);
    if (!slots_ && bytes < kAllocFrom) return plain();
    int device = 0;
    if (!prepare() || cudaGetDevice(&device) != cudaSuccess) return plain();

    const size_t part = (bytes + threads - 1) / threads;
    std::atomic<int> failed{cudaSuccess};
    const auto copy = [&](int t) {
        const size_t begin = std::min(bytes, part * t), count = std::min(bytes, begin + part) - begin;
        const size_t chunks = (count + kChunk - 1) / kChunk;
        char* slot = slots_ + t * kSlots * kChunk;
        cudaEvent_t* done = done_ + t * kSlots;
        const auto length = [&](size_t i) { return std::min(kChunk, count - i * kChunk); };
        const auto fetch = [&](size_t i) {
            cudaError_t err = cudaMemcpyAsync(slot + i % kSlots * kChunk, static_cast<const char*>(src) + begin + i * kChunk,
                                              length(i), cudaMemcpyDeviceToHost, st);
            return err == cudaSuccess ? cudaEventRecord(done[i % kSlots], st) : err;
        };
        cudaError_t err = cudaSetDevice(device);
        for (size_t i = 0; i < std::min<size_t>(kSlots, chunks) && err == cudaSuccess; ++i) err = fetch(i);
        for (size_t i = 0; i < chunks && err == cudaSuccess; ++i) {
            err = cudaEventSynchronize(done[i % kSlots]);
            if (err != cudaSuccess) break;
            std::memcpy(static_cast<char*>(dst) + begin + i * kChunk, slot + i % kSlots * kChunk, length(i));
            if (i + kSlots < chunks) err = fetch(i + kSlots);
        }
        if (err != cudaSuccess) failed = err;
    };
    std::thread helper[kThreads];
    for (int t = 1; t < threads; ++t) {
        try {
            helper[t] = std::thread(copy, t);
        } catch (...) {  // no thread to be had: this one copies the range
            copy(t);
        }
    }
    copy(0);
    for (std::thread& h : helper)
        if (h.joinable()) h.join();
    const cudaError_t err = cudaStreamSynchronize(st);  // nothing in flight when the slots change hands
    return failed != cudaSuccess ? static_cast<cudaError_t>(failed.load()) : err;
}

}  // namespace mpm
