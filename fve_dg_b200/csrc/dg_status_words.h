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

}  // namespace fvedg
