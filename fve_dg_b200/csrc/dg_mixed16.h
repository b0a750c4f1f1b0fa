// Launches of the kernels for groups of sixteen (dg_kernels_mixed16.cuh), compiled in dg_mixed16.cu.
#pragma once
#include <cuda_runtime.h>

#include "dg_kernels_mixed16.cuh"
#include "dg_persistent.h"

namespace fvedg {

// (order, tet rule, tri rule) must be one of FVEDG_MIXED_COMBOS; DG_E_ARG otherwise.
int mixed16_face(int order, int qv, int qf, int sms, const Mixed16FaceArgs& a, cudaStream_t s);
int mixed16_element(int order, int qv, int qf, int sms, const Mixed16ElemArgs& a, cudaStream_t s);
// One stage as a persistent launch over the tile list.
int mixed16_stage(int order, int qv, int qf, int sms, const Mixed16FaceArgs& fa, const Mixed16ElemArgs& ea,
                  const TileQueue& q, cudaStream_t s);
// Warps of the element kernel's CTA (one per SM).
int mixed16_element_warps(int order, int qv, int qf);

}  // namespace fvedg
