// Instances and launches of the FP64 kernels for rows of eight.
#include "dg_fp64_rows.h"

#include <algorithm>

#include "dg_status.cuh"

namespace fvedg {
namespace {

// Resident warps per SM, by the registers a thread needs: sixteen at 128 up to P2 (P1 face kernel 0.090 against
// 0.104 ms with twelve, element kernel 0.077 against 0.090, 196,608 tets), twelve at 168 at P3 (face 0.352 against
// 0.391 ms with eight), eight at 255 above.
constexpr int most_warps(int nb) { return nb <= 10 ? 16 : nb <= 20 ? 12 : 8; }

template <int NB, int NQF>
int run_face(int sms, const Rows8FaceArgs& a, cudaStream_t s) {
    constexpr int W = warps16(most_warps(NB), sizeof(FaceSmem8<NB>));
    constexpr size_t smem = sizeof(FaceSmem8<NB>) * W;
    static unsigned long long done = 0;
    if (const int rc = ensure_smem(face_flux_rows8<NB, NQF, W>, smem, done)) return rc;
    return a.ngroups > 0 ? launch_early(face_flux_rows8<NB, NQF, W>, std::min(a.ngroups, sms), W * 32, smem, s, a) : (int)DG_OK;
}

template <int NB, int NQV>
int run_element(int sms, const Rows8ElemArgs& a, cudaStream_t s) {
    constexpr int W = warps16(most_warps(NB), sizeof(ElemSmem8<NB>));
    constexpr size_t smem = sizeof(ElemSmem8<NB>) * W;
    static unsigned long long done = 0;
    if (const int rc = ensure_smem(element_rows8<NB, NQV, W>, smem, done)) return rc;
    return a.ngroups > 0 ? launch_early(element_rows8<NB, NQV, W>, std::min(a.ngroups, sms), W * 32, smem, s, a) : (int)DG_OK;
}

}  // namespace

int rows8_face(int order, int qv, int qf, int sms, const Rows8FaceArgs& a, cudaStream_t s) {
#define X(P, QV, QF, NB, NQV, NQF) \
    if (order == P && qv == QV && qf == QF) return run_face<NB, NQF>(sms, a, s);
    FVEDG_ROWS8_COMBOS(X)
#undef X
    return DG_E_ARG;
}

int rows8_element(int order, int qv, int qf, int sms, const Rows8ElemArgs& a, cudaStream_t s) {
#define X(P, QV, QF, NB, NQV, NQF) \
    if (order == P && qv == QV && qf == QF) return run_element<NB, NQV>(sms, a, s);
    FVEDG_ROWS8_COMBOS(X)
#undef X
    return DG_E_ARG;
}

}  // namespace fvedg
