// Launches of the viscous (and fused Navier-Stokes) kernels in rows of eight, compiled in dg_viscous_rows.cu.
#pragma once
#include <algorithm>

#include "dg_fp64_rows.h"
#include "dg_viscous_rows.cuh"

namespace fvedg {

// Orders 1..4 of FVEDG_ROWS8_COMBOS; DG_E_ARG otherwise. conv: with the convective terms.
int visc8_face(int order, int qv, int qf, int sms, const Visc8Args& a, bool conv, cudaStream_t s);
int visc8_element(int order, int qv, int qf, int sms, const Visc8Args& a, bool conv, cudaStream_t s);

}  // namespace fvedg
