// Copies between a caller's pageable arrays and the device. The driver stages such a copy through pinned memory with
// one thread, at what one core copies (17 GB/s here, where the link does three times that); large ones are staged by
// several threads instead, each with its own part of the rows and two pinned chunks, so that the link works while the
// cores copy.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <thread>
#include <utility>

#include "dg_status.cuh"

namespace fvedg {

constexpr int kStageThreads = 4;
constexpr size_t kStageChunk = (size_t)1 << 20;
constexpr size_t kStageLeast = (size_t)4 << 20;  // bytes from which the threads pay for themselves

struct StageBlock {
    enum State { kAbsent, kIdle, kBusy };
    State state = kAbsent;
    char* mem = nullptr;  // [kStageThreads][2][kStageChunk], pinned
    cudaEvent_t ev[kStageThreads][2] = {};
};

// Pinned blocks, shared by all contexts: a transfer takes one for its duration. A device has at most two, idle ones
// among them, and none once the last context is gone. A third transfer at the same time is the driver's: with a block of
// its own, made and freed by each call, six threads took 1,429 us for 5.3 MB in and out (415 without any block). No call
// allocates from the heap, so that none can throw.
class StagePool {
  public:
    static StagePool& get() {
        static StagePool p;  // nothing to destroy: it outlives every context, also those that a program never closes
        return p;
    }
    void open() {
        std::lock_guard<std::mutex> g(m_);
        ++contexts_;
    }
    void close() {
        StageBlock gone[kDevices][kBlocks];
        {
            std::lock_guard<std::mutex> g(m_);
            if (--contexts_ > 0) return;
            for (int d = 0; d < kDevices; ++d)
                for (int i = 0; i < kBlocks; ++i)
                    if (block_[d][i].state == StageBlock::kIdle) std::swap(gone[d][i], block_[d][i]);
        }
        for (auto& of_device : gone)
            for (StageBlock& b : of_device) destroy(b);
    }
    // A block of the device, or null: both are taken, or there is no memory for one.
    StageBlock* take(int device) {
        if (device < 0 || device >= kDevices) return nullptr;
        StageBlock* b = nullptr;
        {
            std::lock_guard<std::mutex> g(m_);
            for (StageBlock& x : block_[device])
                if (x.state != StageBlock::kBusy && (!b || x.state == StageBlock::kIdle)) b = &x;
            if (!b) return nullptr;
            b->state = StageBlock::kBusy;
            if (b->mem) return b;
        }
        bool ok = cudaHostAlloc((void**)&b->mem, kStageThreads * 2 * kStageChunk, cudaHostAllocPortable) == cudaSuccess;
        for (auto& e : b->ev)
            for (cudaEvent_t& x : e) ok = ok && cudaEventCreateWithFlags(&x, cudaEventDisableTiming) == cudaSuccess;
        if (ok) return b;
        cudaGetLastError();
        give(b, false);
        return nullptr;
    }
    void give(StageBlock* b, bool keep = true) {
        StageBlock gone;
        {
            std::lock_guard<std::mutex> g(m_);
            b->state = StageBlock::kIdle;
            if (!keep || contexts_ == 0) std::swap(gone, *b);
        }
        destroy(gone);
    }

  private:
    static constexpr int kDevices = 16, kBlocks = 2;
    static void destroy(StageBlock& b) {
        for (auto& e : b.ev)
            for (cudaEvent_t x : e)
                if (x) {
                    cudaEventSynchronize(x);
                    cudaEventDestroy(x);
                }
        if (b.mem) cudaFreeHost(b.mem);
    }
    std::mutex m_;
    StageBlock block_[kDevices][kBlocks];
    int contexts_ = 0;
};

// A context's share in the pool's life.
struct StageUse {
    StageUse() { StagePool::get().open(); }
    ~StageUse() { StagePool::get().close(); }
    StageUse(const StageUse&) = delete;
    StageUse& operator=(const StageUse&) = delete;
};

// Whether rows of `blk` bytes at `host` are copied by staged_copy: large, and pageable memory.
inline bool staged(const void* host, size_t blk, int64_t nrow) {
    if (blk * (size_t)nrow < kStageLeast || blk > kStageChunk || std::thread::hardware_concurrency() < 4) return false;
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// Rows [0, nrow) of `blk` bytes, `stride` apart on the host and packed on the device, on stream s. On return the host
// array has been read (to the device) or written (from it). 1: no block to be had, nothing done.
inline int staged_copy(bool to_device, char* dev, char* host, size_t stride, size_t blk, int64_t nrow, int device, cudaStream_t s) {
    StageBlock* const block = StagePool::get().take(device);
    if (!block) return 1;
    StageBlock& b = *block;
    const int64_t per = (int64_t)(kStageChunk / blk);  // rows of a chunk
    auto rows = [&](char* pinned, int64_t r0, int64_t n) {
        char* h = host + r0 * stride;
        if (stride == blk) {
            if (to_device) memcpy(pinned, h, n * blk);
            else memcpy(h, pinned, n * blk);
            return;
        }
        for (int64_t i = 0; i < n; ++i) {
            if (to_device) memcpy(pinned + i * blk, h + i * stride, blk);
            else memcpy(h + i * stride, pinned + i * blk, blk);
        }
    };
    auto part = [&](int t) -> cudaError_t {
        cudaError_t rc = cudaSetDevice(device);
        const int64_t lo = nrow * t / kStageThreads, hi = nrow * (t + 1) / kStageThreads;
        const int64_t nchunk = (hi - lo + per - 1) / per;
        char* pinned = b.mem + (size_t)t * 2 * kStageChunk;
        auto send = [&](int64_t j) {  // chunk j across the link
            const int64_t r0 = lo + j * per, n = std::min(per, hi - r0);
            char *d = dev + r0 * blk, *p = pinned + (j & 1) * kStageChunk;
            cudaError_t e = to_device ? cudaMemcpyAsync(d, p, n * blk, cudaMemcpyHostToDevice, s)
                                      : cudaMemcpyAsync(p, d, n * blk, cudaMemcpyDeviceToHost, s);
            return e == cudaSuccess ? cudaEventRecord(b.ev[t][j & 1], s) : e;
        };
        // a chunk's event is that of the last copy from or to it, possibly an earlier transfer's to the device
        if (!to_device)
            for (int64_t j = 0; j < std::min<int64_t>(2, nchunk) && rc == cudaSuccess; ++j)
                if ((rc = cudaEventSynchronize(b.ev[t][j])) == cudaSuccess) rc = send(j);
        for (int64_t j = 0; j < nchunk && rc == cudaSuccess; ++j) {
            const int64_t r0 = lo + j * per, n = std::min(per, hi - r0);
            char* p = pinned + (j & 1) * kStageChunk;
            if ((rc = cudaEventSynchronize(b.ev[t][j & 1])) != cudaSuccess) break;
            rows(p, r0, n);
            if (to_device) rc = send(j);
            else if (j + 2 < nchunk) rc = send(j + 2);
        }
        return rc;
    };
    cudaError_t rc[kStageThreads] = {};
    std::thread helper[kStageThreads];
    for (int t = 1; t < kStageThreads; ++t) {
        try {
            helper[t] = std::thread([&, t] { rc[t] = part(t); });
        } catch (...) {  // no thread, or no memory for one: its part is done here
        }
    }
    rc[0] = part(0);
    for (int t = 1; t < kStageThreads; ++t) {
        if (helper[t].joinable()) helper[t].join();
        else rc[t] = part(t);
    }
    int out = DG_OK;
    for (cudaError_t e : rc)
        if (e != cudaSuccess) out = cuda_status(e);
    StagePool::get().give(block);
    return out;
}

}  // namespace fvedg
