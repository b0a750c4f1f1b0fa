// Instances and launches of the viscous and Navier-Stokes kernels in rows of eight.
#include "dg_viscous_rows.h"

#include "dg_status.cuh"

namespace fvedg {
namespace {

// Eight warps per SM at 255 registers a thread, twelve at P1.
constexpr int most_warps(int nb) { return nb <= 4 ? 12 : 8; }

template <int NB, int NQF, bool CONV>
int run_face(int sms, const Visc8Args& a, cudaStream_t s) {
    constexpr int W = warps16(most_warps(NB), sizeof(FaceSmem8<NB>));
    constexpr size_t smem = sizeof(FaceSmem8<NB>) * W;
    static unsigned long long done = 0;
    if (const int rc = ensure_smem(visc_face_rows8<NB, NQF, CONV, W>, smem, done)) return rc;
    return a.f.ngroups > 0 ? launch_early(visc_face_rows8<NB, NQF, CONV, W>, std::min(a.f.ngroups, sms), W * 32, smem, s, a) : (int)DG_OK;
}

template <int NB, int NQV, bool CONV>
int run_element(int sms, const Visc8Args& a, cudaStream_t s) {
    constexpr int W = warps16(most_warps(NB), sizeof(ElemSmem8<NB>));
    constexpr size_t smem = sizeof(ElemSmem8<NB>) * W;
    static unsigned long long done = 0;
    if (const int rc = ensure_smem(visc_element_rows8<NB, NQV, CONV, W>, smem, done)) return rc;
    return a.e.ngroups > 0 ? launch_early(visc_element_rows8<NB, NQV, CONV, W>, std::min(a.e.ngroups, sms), W * 32, smem, s, a) : (int)DG_OK;
}

}  // namespace

int visc8_face(int order, int qv, int qf, int sms, const Visc8Args& a, bool conv, cudaStream_t s) {
#define X(P, QV, QF, NB, NQV, NQF)                                                                          \
    if constexpr (P >= 1 && P <= 4)                                                                         \
        if (order == P && qv == QV && qf == QF)                                                             \
            return conv ? run_face<NB, NQF, true>(sms, a, s) : run_face<NB, NQF, false>(sms, a, s);
    FVEDG_ROWS8_COMBOS(X)
#undef X
    return DG_E_ARG;
}

int visc8_element(int order, int qv, int qf, int sms, const Visc8Args& a, bool conv, cudaStream_t s) {
#define X(P, QV, QF, NB, NQV, NQF)                                                                          \
    if constexpr (P >= 1 && P <= 4)                                                                         \
        if (order == P && qv == QV && qf == QF)                                                             \
            return conv ? run_element<NB, NQV, true>(sms, a, s) : run_element<NB, NQV, false>(sms, a, s);
    FVEDG_ROWS8_COMBOS(X)
#undef X
    return DG_E_ARG;
}

}  // namespace fvedg
