// Rule combinations of the mixed-precision form.
#pragma once

// X(order, qv, qf, NB, NQV, NQF, W): W warps per block of the element kernel
#define FVEDG_MIXED_COMBOS(X)      \
    X(1, 0, 1, 4, 4, 6, 8)         \
    X(1, 0, 0, 4, 4, 4, 8)         \
    X(1, 0, 2, 4, 4, 7, 8)         \
    X(1, 2, 2, 4, 15, 7, 8)        \
    X(2, 1, 2, 10, 11, 7, 8)       \
    X(2, 1, 3, 10, 11, 24, 8)      \
    X(2, 2, 3, 10, 15, 24, 8)      \
    X(3, 3, 3, 20, 23, 24, 8)      \
    X(3, 4, 3, 20, 31, 24, 8)      \
    X(4, 5, 3, 35, 44, 24, 4)      \
    X(4, 6, 3, 35, 57, 24, 4)
