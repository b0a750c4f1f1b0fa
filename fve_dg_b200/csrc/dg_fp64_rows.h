// Launches of the FP64 kernels for rows of eight (dg_kernels_fp64_rows.cuh), compiled in dg_fp64_rows.cu.
#pragma once
#include <cuda_runtime.h>

#include "dg_kernels_fp64_rows.cuh"

namespace fvedg {

// (order, tet rule, tri rule) combinations with these kernels: X(P, QV, QF, NB, NQV, NQF)
#define FVEDG_ROWS8_COMBOS(X) \
    X(0, 2, 2, 1, 15, 7)      \
    X(1, 0, 1, 4, 4, 6)       \
    X(1, 0, 0, 4, 4, 4)       \
    X(1, 0, 2, 4, 4, 7)       \
    X(1, 2, 2, 4, 15, 7)      \
    X(2, 1, 2, 10, 11, 7)     \
    X(2, 1, 3, 10, 11, 24)    \
    X(2, 2, 3, 10, 15, 24)    \
    X(3, 3, 3, 20, 23, 24)    \
    X(3, 4, 3, 20, 31, 24)    \
    X(4, 5, 3, 35, 44, 24)    \
    X(4, 6, 3, 35, 57, 24)    \
    X(5, 7, 4, 56, 94, 36)

int rows8_face(int order, int qv, int qf, int sms, const Rows8FaceArgs& a, cudaStream_t s);
int rows8_element(int order, int qv, int qf, int sms, const Rows8ElemArgs& a, cudaStream_t s);

}  // namespace fvedg
