// Status words of the kernels' bounded waits, in mapped host memory: the host reads them after a synchronize without a
// copy. Pages of them are shared by the contexts (a mapping costs two to three milliseconds), so that there are at most
// as many as the most contexts alive at once need, 256 to a page.
#pragma once
#include <cuda_runtime.h>

#include <mutex>
#include <new>

#include "dg_gpu.h"

namespace fvedg {

constexpr int kStatusWords = 4;  // of a context: mixed kernels, rows of eight, viscous ones, spare

class StatusPages {
  public:
    static StatusPages& get() {
        static StatusPages* p = new StatusPages;  // outlives every context, also those that a program never closes
        return *p;
    }
    // A context's words, DG_OK; null without memory for them.
    int* take() {
        std::lock_guard<std::mutex> g(m_);
        for (Page* p = first_;; p = p->next) {
            if (!p) {
                p = new (std::nothrow) Page;
                if (!p) return nullptr;
                if (cudaHostAlloc((void**)&p->words, sizeof(int) * kStatusWords * kSlots, cudaHostAllocMapped | cudaHostAllocPortable) !=
                    cudaSuccess) {
                    delete p;
                    return nullptr;
                }
                p->next = first_;
                first_ = p;
            }
            for (int i = 0; i < kSlots; ++i)
                if (!p->used[i]) {
                    p->used[i] = true;
                    int* w = p->words + kStatusWords * i;
                    for (int k = 0; k < kStatusWords; ++k) w[k] = DG_OK;
                    return w;
                }
        }
    }
    void give(const int* w) {
        std::lock_guard<std::mutex> g(m_);
        for (Page* p = first_; p; p = p->next)
            if (w >= p->words && w < p->words + kStatusWords * kSlots) p->used[(w - p->words) / kStatusWords] = false;
    }

  private:
    static constexpr int kSlots = 256;
    struct Page {
        int* words = nullptr;
        bool used[kSlots] = {};
        Page* next = nullptr;
    };
    std::mutex m_;
    Page* first_ = nullptr;
};

// After a synchronize: DG_OK, or DG_E_WATCHDOG if a bounded wait ran out; the words are cleared. They lie in mapped host
// memory: read by copies from the device they were 8 us of every stepping call.
inline int take_status(int* words) {
    int rc = DG_OK;
    for (int i = 0; i < kStatusWords; ++i) {
        volatile int* word = words + i;
        if (*word == DG_OK) continue;
        *word = DG_OK;
        rc = DG_E_WATCHDOG;
    }
    return rc;
}

// The same with a tile queue's own error, which `read` fetches and `clear` re-arms (DG_OK or their own failure). Either is
// taken whatever the other says: nothing that this call reports is left for the next.
template <class Read, class Clear>
int take_status(int* words, Read&& read, Clear&& clear) {
    const int rc = take_status(words);
    int error = DG_OK;
    if (const int failed = read(&error)) return failed;
    if (error == DG_OK) return rc;
    if (const int failed = clear()) return failed;
    return DG_E_WATCHDOG;
}

}  // namespace fvedg
