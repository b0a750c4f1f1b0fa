// The tile queue of the persistent schedule: what its kernels share (dg_persistent.cuh says how it works).
#pragma once
#include <cuda_runtime.h>

#include "dg_gpu.h"

namespace fvedg {

constexpr int kMaxRegions = 64;

struct QueueState {
    unsigned int ticket;              // next tile of the list
    unsigned int exits;               // CTAs that have left this launch
    int error;                        // DG_OK or DG_E_WATCHDOG
    int pad;
    unsigned int done[kMaxRegions];   // face groups completed, per region
};

struct TileQueue {
    QueueState* q;
    const int4* tiles;                // {kind (0 face, 1 element), first group, end group, region}
    int ntiles;
    const unsigned long long* deps;   // [R] face regions each element region reads
    const unsigned int* total;        // [R] face groups per region
    long long spin_limit;             // polls before a wait gives up
};

#ifdef __CUDACC__
// Thread 0 of the CTA takes the next tile ({-1, ...} past the end) and, for an element tile, waits until the
// face regions it reads are complete (bounded; an expired wait is recorded and the tile goes on).
__device__ __forceinline__ int4 take_tile(const TileQueue& Q) {
    const unsigned int t = atomicAdd(&Q.q->ticket, 1u);
    const int4 tl = t < (unsigned int)Q.ntiles ? Q.tiles[t] : make_int4(-1, 0, 0, 0);
    if (tl.x == 1) {
        unsigned long long need = Q.deps[tl.w];
        while (need) {
            const int f = __ffsll((long long)need) - 1;
            const volatile unsigned int* d = &Q.q->done[f];
            long long spins = 0;
            while (*d < Q.total[f]) {
                __nanosleep(64);
                if (++spins > Q.spin_limit) {
                    atomicExch(&Q.q->error, DG_E_WATCHDOG);
                    break;
                }
            }
            need &= need - 1;
        }
        __threadfence();
    }
    return tl;
}

// Thread 0, leaving: the last CTA out re-arms the queue for the next launch.
__device__ __forceinline__ void leave_queue(const TileQueue& Q) {
    __threadfence();
    if (atomicAdd(&Q.q->exits, 1u) == gridDim.x - 1) {
        Q.q->ticket = 0u;
        for (int r = 0; r < kMaxRegions; ++r) Q.q->done[r] = 0u;
        __threadfence();
        Q.q->exits = 0u;
    }
}
#endif

}  // namespace fvedg
