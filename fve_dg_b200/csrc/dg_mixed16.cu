// Instances and launches of the mixed-precision kernels for groups of sixteen.
#include "dg_mixed16.h"

#include <algorithm>

#include "dg_mixed_combos.h"
#include "dg_status.cuh"

namespace fvedg {
namespace {

// Persistent form of a stage: CTAs take face and element tiles of the list (dg_persistent.cuh); every warp
// has one area of shared memory that serves both kinds.
template <int NB, int NQV, int NQF>
__host__ __device__ constexpr size_t stage_warp_smem() {
    constexpr size_t a = sizeof(FaceSmem16<NB, NQF>), b = sizeof(ElemSmem16<NB, NQV>);
    return a > b ? a : b;
}

template <int NB, int NQV, int NQF, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 1) stage_persistent_mixed16(Mixed16FaceArgs fa, Mixed16ElemArgs ea, TileQueue Q) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint64_t bars[WARPS];
    __shared__ int4 s_tile;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const ElemTables16 t = elem_tables16<NB, NQV>(ea.t, smem_raw);
    unsigned char* mine = smem_raw + ElemSizes16<NB, NQV>::tables + stage_warp_smem<NB, NQV, NQF>() * warp;
    if (lane == 0) mbar_init(&bars[warp], kRows);
    unsigned parity = 0;
    bool ok = true;  // a warp whose copies did not land does no further groups
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_tile = take_tile(Q);
        __syncthreads();
        const int4 tl = s_tile;
        if (tl.x < 0) break;
        if (tl.x == 0) {
            if (ok) ok = face_run16<NB, NQF>(fa, tl.y + warp, tl.z, WARPS, *reinterpret_cast<FaceSmem16<NB, NQF>*>(mine),
                                             bars[warp], parity, lane);
            __threadfence();  // this CTA's records are visible before the region count moves
            __syncthreads();
            if (threadIdx.x == 0) atomicAdd(&Q.q->done[tl.w], (unsigned int)(tl.z - tl.y));
        } else if (ok) {
            ok = elem_run16<NB, NQV>(ea, t, tl.y + warp, tl.z, WARPS, *reinterpret_cast<ElemSmem16<NB, NQV>*>(mine),
                                     bars[warp], parity, lane);
        }
    }
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    if (threadIdx.x == 0) leave_queue(Q);
}

// Resident warps per SM: twelve at 168 registers a thread where that is enough, else eight at 255.
template <int NB, int NQF>
constexpr int face_warps() { return warps16(NB <= 20 ? 12 : 8, sizeof(FaceSmem16<NB, NQF>)); }
template <int NB, int NQV>
constexpr int element_warps() {
    return warps16(NB <= 10 ? 12 : 8, sizeof(ElemSmem16<NB, NQV>), ElemSizes16<NB, NQV>::tables);
}

template <int NB, int NQF>
int run_face(int sms, const Mixed16FaceArgs& a, cudaStream_t s) {
    constexpr int W = face_warps<NB, NQF>();
    constexpr size_t smem = sizeof(FaceSmem16<NB, NQF>) * W;
    static unsigned long long done = 0;
    if (const int rc = ensure_smem(face_flux_mixed16<NB, NQF, W>, smem, done)) return rc;
    return a.ngroups > 0 ? launch_early(face_flux_mixed16<NB, NQF, W>, std::min((a.ngroups + W - 1) / W, sms), W * 32, smem, s, a) : (int)DG_OK;
}

template <int NB, int NQV>
int run_element(int sms, const Mixed16ElemArgs& a, cudaStream_t s) {
    constexpr int W = element_warps<NB, NQV>();
    constexpr size_t smem = ElemSizes16<NB, NQV>::tables + sizeof(ElemSmem16<NB, NQV>) * W;
    static unsigned long long done = 0;
    if (const int rc = ensure_smem(element_mixed16<NB, NQV, W>, smem, done)) return rc;
    return a.ngroups > 0 ? launch_early(element_mixed16<NB, NQV, W>, std::min((a.ngroups + W - 1) / W, sms), W * 32, smem, s, a) : (int)DG_OK;
}

template <int NB, int NQV, int NQF>
int run_stage(int sms, const Mixed16FaceArgs& fa, const Mixed16ElemArgs& ea, const TileQueue& q, cudaStream_t s) {
    constexpr size_t tables = ElemSizes16<NB, NQV>::tables, warp = stage_warp_smem<NB, NQV, NQF>();
    constexpr int W = warps16(NB <= 10 ? 12 : 8, warp, tables);
    constexpr size_t smem = tables + warp * W;
    static unsigned long long done = 0;
    if (const int rc = ensure_smem(stage_persistent_mixed16<NB, NQV, NQF, W>, smem, done)) return rc;
    stage_persistent_mixed16<NB, NQV, NQF, W><<<sms, W * 32, smem, s>>>(fa, ea, q);
    return cuda_status(cudaGetLastError());
}

}  // namespace

int mixed16_face(int order, int qv, int qf, int sms, const Mixed16FaceArgs& a, cudaStream_t s) {
#define X(P, QV, QF, NB, NQV, NQF, W) \
    if (order == P && qv == QV && qf == QF) return run_face<NB, NQF>(sms, a, s);
    FVEDG_MIXED_COMBOS(X)
#undef X
    return DG_E_ARG;
}

int mixed16_element(int order, int qv, int qf, int sms, const Mixed16ElemArgs& a, cudaStream_t s) {
#define X(P, QV, QF, NB, NQV, NQF, W) \
    if (order == P && qv == QV && qf == QF) return run_element<NB, NQV>(sms, a, s);
    FVEDG_MIXED_COMBOS(X)
#undef X
    return DG_E_ARG;
}

int mixed16_stage(int order, int qv, int qf, int sms, const Mixed16FaceArgs& fa, const Mixed16ElemArgs& ea,
                  const TileQueue& q, cudaStream_t s) {
#define X(P, QV, QF, NB, NQV, NQF, W) \
    if (order == P && qv == QV && qf == QF) return run_stage<NB, NQV, NQF>(sms, fa, ea, q, s);
    FVEDG_MIXED_COMBOS(X)
#undef X
    return DG_E_ARG;
}

int mixed16_element_warps(int order, int qv, int qf) {
#define X(P, QV, QF, NB, NQV, NQF, W) \
    if (order == P && qv == QV && qf == QF) return element_warps<NB, NQV>();
    FVEDG_MIXED_COMBOS(X)
#undef X
    return 0;
}

}  // namespace fvedg
