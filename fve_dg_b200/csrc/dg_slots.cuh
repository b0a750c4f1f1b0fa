// State rows in shared memory, moved by TMA bulk copies on a warp's own mbarrier.
#pragma once
#include "dg_gpu.h"
#include "dg_tma.cuh"

namespace fvedg {

// One slot per item, BYTES apart. A row that starts on an 8-byte boundary keeps that offset in its slot, so
// that its middle is one bulk copy (16-byte aligned on both sides) whatever the row length; a first or last
// double that sticks out is moved by itself.
template <int NB, int STRIDE>
struct RowSlotsOf {
    static constexpr int LEN = 5 * NB, BYTES = STRIDE;
    static_assert(STRIDE % 16 == 0 && STRIDE >= 8 * LEN + 8, "a row and its offset");
    static __device__ __forceinline__ int skew(const double* row) { return (int)(reinterpret_cast<uintptr_t>(row) & 8); }
    static __device__ __forceinline__ double* at(void* slots, int i, const double* row) {
        return reinterpret_cast<double*>(static_cast<char*>(slots) + i * BYTES + skew(row));
    }
    // Lane `lane` < n: its row into slot `lane`; every such lane announces its own bytes on `bar` (count n).
    static __device__ __forceinline__ void load(void* slots, int lane, int n, const double* row, uint64_t* bar) {
        if (lane < n) {
            double* to = at(slots, lane, row);
            const int head = skew(row) ? 1 : 0, mid = (LEN - head) & ~1, tail = LEN - head - mid;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            if (LEN % 2 == 0 && !head) {
                mbar_arrive_expect_tx(bar, 8u * LEN);
                bulk_copy_g2s(to, row, 8u * LEN, bar);
            } else {  // the arrival follows the stores of this lane, which it releases
                mbar_expect_tx(bar, 8u * mid);
                bulk_copy_g2s(to + head, row + head, 8u * mid, bar);
                if (head) to[0] = row[0];
                if (tail) to[LEN - 1] = row[LEN - 1];
                mbar_arrive(bar);
            }
        }
    }
    // Lane `lane` < n: slot `lane` back to its row; the caller has fenced the slots' writes.
    static __device__ __forceinline__ void store(void* slots, int lane, int n, double* row) {
        if (lane < n) {
            double* from = at(slots, lane, row);
            const int head = skew(row) ? 1 : 0, mid = (LEN - head) & ~1, tail = LEN - head - mid;
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(row + head),
                         "r"(smem_addr(from + head)), "r"(8u * mid)
                         : "memory");
            if (head) row[0] = from[0];
            if (tail) row[LEN - 1] = from[LEN - 1];
        }
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
};

// The whole warp waits for phase `parity` of its barrier, a bounded number of polls. If they run out for any lane, that is
// recorded, the copies in flight are let in (bounded again) and every lane has false, also one that saw them land in its
// last poll. The vote comes before the branch or after it, whichever the kernel is faster with (us, after / before): groups
// of sixteen P2, four steps of 196,608 cells 2,856 / 2,816, P4, 93,750 cells 5,292 / 5,247, the persistent form 5,665 / 5,572;
// the viscous kernels, a Navier-Stokes step at P3, 82,944 cells 1,931 / 1,922. But groups of eight, a residual, P2, 13,182 cells 32.7 / 33.0, P5, 7,986 cells 220 / 227.
template <bool VOTE_FIRST>
__device__ __forceinline__ bool warp_landed(uint64_t* bar, unsigned parity, int* err) {
    bool ok = mbar_wait_bounded(bar, parity, kBulkSpinLimit);
    if constexpr (VOTE_FIRST) ok = __all_sync(0xffffffffu, ok);
    if (!ok) {
        if (err) *static_cast<volatile int*>(err) = DG_E_WATCHDOG;
        mbar_wait_bounded(bar, parity, kBulkSpinLimit);
    }
    if constexpr (!VOTE_FIRST) ok = __all_sync(0xffffffffu, ok);
    return ok;
}

// The same for the warp's rows, whose barrier is in its next phase afterwards.
template <bool VOTE_FIRST = false>
__device__ __forceinline__ bool rows_landed(uint64_t& bar, unsigned& parity, int* err) {
    const bool ok = warp_landed<VOTE_FIRST>(&bar, parity, err);
    parity ^= 1u;
    return ok;
}

}  // namespace fvedg
