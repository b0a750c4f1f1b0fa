// Positivity-preserving two-step limiter, after include/DG/DG_Schemes/PositiveLimiter.h:12-261, as
// the reference's drivers call it: constructMinMax(current, previous) then apply(current, previous)
// (examples/Eular1D/Sod1D/Riemann1D.cpp:194-195). FP64 in both forms.
//
//   bounds (constructMinMax, :57-103): per face, both cells' previous states evaluated at the
//     volume rule's reference points; max over points of max(v1, v2) per variable, and - as the
//     reference computes it (:86) - the min is min(v1, v2) at the last point. With only_avg the
//     bounds are the max/min of the two cells' means. A boundary face uses its one cell twice.
//     Each cell's bounds are the max/min over its faces.
//   step 1 (apply_1_limitCell, :128-163): per variable, if the quadrature values leave the cell's
//     bounds, scale the modes l >= 1 by min(theta_min, theta_max, 1) with
//     theta_min = (avg - min_b) / (avg - v_min + 1e-32), theta_max = (max_b - avg) / (v_max - avg + 1e-32).
//   step 2 (apply_21_limitCell, :164-188): density kept >= 1e-16 at the points by scaling its modes.
//   step 3 (apply_22_limitCell, :189-258): for every point with negative pressure, 100 bisection
//     steps on t in [0, 1] for p((1 - t) avg + t U(x_g)) = 0; all modes l >= 1 scaled by the
//     smallest t.
// Means are never changed, so mass, momentum and energy are conserved exactly.
//
// Per-cell statistics of the previous state (lanes over the quadrature points, each point value summed
// over the modes in order, as the reference does), then the bounds and the three steps with the cells
// of a warp side by side. In the time loop the statistics of each stage's limited output come out of
// the same launch and bound the next stage, so one launch per stage suffices. Warps never wait on one
// another.
#pragma once
#include <cfloat>

#include "dg_kernels_fp64.cuh"
#include "dg_launch.cuh"
#include "dg_status.cuh"
#include "dg_mixed_host.cuh"

namespace fvedg {

__device__ __forceinline__ double ref_max(double a, double b) { return (a < b) ? b : a; }  // std::max
__device__ __forceinline__ double ref_min(double a, double b) { return (b < a) ? b : a; }  // std::min

__device__ __forceinline__ double warp_max(double v) {
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = ref_max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ double warp_min(double v) {
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = ref_min(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// PositiveLimiter.h:112-123
__device__ __forceinline__ double limiter_pressure(const double U[5], double gamma) {
    const double rho = U[0];
    if (rho <= 1e-16) return -1.0;
    const double ke = (U[1] * U[1] + U[2] * U[2] + U[3] * U[3]) / (2.0 * rho);
    return (gamma - 1.0) * (U[4] - ke);
}

// limiter_pressure(U, gamma) < 0, without the division where the sign is clear of rounding: E (2 rho) against m^2,
// a hundred units in the last place apart, and nothing near underflow.
__device__ __forceinline__ bool negative_pressure(const double U[5], double gamma) {
    const double rho = U[0];
    if (rho <= 1e-16) return true;
    const double m2 = U[1] * U[1] + U[2] * U[2] + U[3] * U[3], t = U[4] * (2.0 * rho);
    if (gamma > 1.001) {
        if (t > m2 * (1.0 + 1e-14) && t > 1e-80) return false;
        if (t < m2 * (1.0 - 1e-14) && m2 > 1e-100 && rho < 1e100) return true;
    }
    return limiter_pressure(U, gamma) < 0;
}

constexpr int kLimWarps = 4;       // statistics alone
constexpr int kLimApplyWarps = 8;  // the three steps, two blocks per SM

// The volume rule's basis values transposed to [l][g] in shared memory: lanes over points read
// consecutive doubles (conflict-free) for every mode l.
template <int NB, int NQV>
__device__ __forceinline__ void load_phi_t(double* sphi, const double* __restrict__ phi) {
    for (int i = threadIdx.x; i < NQV * NB; i += blockDim.x) {
        const int g = i / NB, l = i - g * NB;
        sphi[l * NQV + g] = phi[i];
    }
}

// The 5 conserved values at volume point g from the transposed table, summed over the modes in
// order, as the reference evaluates a point value.
template <int NB, int NQV>
__device__ __forceinline__ void point_values_t(const double* sphi, const double* u, int g, double v[5]) {
    #pragma unroll
    for (int k = 0; k < 5; ++k) v[k] = 0.0;
    #pragma unroll 4
    for (int l = 0; l < NB; ++l) {
        const double p = sphi[l * NQV + g];
        #pragma unroll
        for (int k = 0; k < 5; ++k) v[k] = fma(p, u[k + 5 * l], v[k]);
    }
}

// Lanes per cell in the apply pass: the cells of a warp are processed side by side by groups of G
// lanes (G a power of two), each lane holding ceil(NQV / G) points. Few lanes: what a cell's lanes do alike (bounds,
// reductions) is then shared by more cells of a warp instruction; as many as keep the points in registers.
template <int NQV>
struct LimGroup {
    static constexpr int G = NQV <= 24 ? 4 : NQV <= 48 ? 8 : 16;
};

template <int G>
__device__ __forceinline__ double group_max(double v, unsigned mask) {
    #pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v = ref_max(v, __shfl_xor_sync(mask, v, o));
    return v;
}
template <int G>
__device__ __forceinline__ double group_min(double v, unsigned mask) {
    #pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) v = ref_min(v, __shfl_xor_sync(mask, v, o));
    return v;
}

// A cell's statistics from its point values v[PPL][5], held by a group of G lanes (lane gl holds
// points gl + G r): the max over the points of each variable and the values at the last point
// (with only_avg: the mean, twice).
template <int NQV, int G, int PPL>
__device__ __forceinline__ void write_stats(const double (&v)[PPL][5], const double (&avg)[5], int gl, unsigned mask,
                                            int only_avg, double* out, bool live = true) {
    if (only_avg) {
        #pragma unroll
        for (int k = 0; k < 5; ++k)
            if (live && gl == k % G) { out[k] = avg[k]; out[5 + k] = avg[k]; }
        return;
    }
    constexpr int LR = (NQV - 1) / G, LL = (NQV - 1) % G;
    if (live && gl == LL) {
        #pragma unroll
        for (int k = 0; k < 5; ++k) out[5 + k] = v[LR][k];
    }
    #pragma unroll
    for (int k = 0; k < 5; ++k) {
        double mx = -DBL_MAX;
        #pragma unroll
        for (int r = 0; r < PPL; ++r)
            if (gl + G * r < NQV) mx = ref_max(mx, v[r][k]);
        mx = group_max<G>(mx, mask);
        if (live && gl == 0) out[k] = mx;
    }
}

// Per-cell statistics of a state for the bounds, cells [c_begin, c_end): the max over the volume
// points of each variable and the values at the last point. A face's bounds are max(v1, v2) over the
// points and min(v1, v2) at the last point (PositiveLimiter.h:77-88), i.e. the max of its two cells'
// maxima and the min of their last-point values; with only_avg both are the cell mean (:70-75).
template <int NB, int NQV>
__global__ void __launch_bounds__(kLimWarps * 32)
    limiter_cell_stats(const double* __restrict__ Up, const double* __restrict__ phi, int64_t c_begin, int64_t c_end,
                       int only_avg, double* __restrict__ stats) {
    constexpr int PPL = (NQV + 31) / 32;
    __shared__ double sphi[NQV * NB];
    __shared__ double scoef[kLimWarps][5 * NB];
    load_phi_t<NB, NQV>(sphi, phi);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    double* u = scoef[threadIdx.x >> 5];
    for (int64_t c = c_begin + (int64_t)blockIdx.x * kLimWarps + (threadIdx.x >> 5); c < c_end;
         c += (int64_t)gridDim.x * kLimWarps) {
        const double* ug = Up + c * (5 * NB);
        for (int i = lane; i < 5 * NB; i += 32) u[i] = ug[i];  // coalesced, then broadcast reads
        __syncwarp();
        double avg[5], v[PPL][5];
        #pragma unroll
        for (int k = 0; k < 5; ++k) avg[k] = u[k];
        if (!only_avg) {
            #pragma unroll
            for (int r = 0; r < PPL; ++r) {
                const int g = lane + 32 * r;
                if (g < NQV) point_values_t<NB, NQV>(sphi, u, g, v[r]);
            }
        }
        write_stats<NQV, 32, PPL>(v, avg, lane, 0xffffffffu, only_avg, stats + c * 10);
        __syncwarp();
    }
}

// Shared memory of limiter_apply: the basis [mode][point], padded to G lanes x PPL points with zeros; per warp two
// buffers of its cells' rows, and the scales of its cells' variables.
template <int NB, int NQV>
struct LimSizes {
    static constexpr int G = LimGroup<NQV>::G, CPW = 32 / G, PPL = (NQV + G - 1) / G, GP = G * PPL;
    static constexpr int CHUNK = CPW * 5 * NB;  // doubles
    static constexpr size_t smem = sizeof(double) * (NB * GP + (kLimApplyWarps * (2 * CHUNK + CPW * 6)));
};

// (avg - min_b) / (avg - v_min + 1e-32) and its counterpart, at most 1 (PositiveLimiter.h:140-160)
__device__ __forceinline__ double limiter_theta(double avg, double vmin, double vmax, double bmin, double bmax) {
    const double tmin = (avg != vmin) ? (avg - bmin) / (avg - vmin + 1e-32) : 0.0;
    const double tmax = (avg != vmax) ? (bmax - avg) / (vmax - avg + 1e-32) : 0.0;
    return ref_min(ref_min(tmin, tmax), 1.0);
}

// The three steps per element (PositiveLimiter.h:128-258) for cells [0, ncell), CPW = 32 / G cells
// per warp side by side (lanes over the points of their cell). Bounds: the max of the statistics'
// maxima and the min of their last-point values over the cell and its face neighbours (nbr
// [ncell][4], the cell itself across a boundary face), which is the max/min over the cell's faces of
// the face bounds: lane i of a cell loads neighbour i's. Point values are evaluated once; after a
// step scales the modes l >= 1 of a variable by theta, its point values become avg + theta (v - avg)
// (phi_0 = 1), which is what the reference re-evaluates. stats_out: when non-null, the statistics of
// the limited state (as limiter_cell_stats computes them: re-evaluated from the new coefficients
// where the limiter acted), the next stage's bounds.
//
// All lanes stay together: a lane group without a cell repeats the warp's last one and stores nothing. Bound by
// instruction issue and the chains within a cell, so: rows arrive two groups of cells ahead, in one piece per
// warp; reductions and divisions of the five variables run side by side, one variable's quotients per lane; the
// sign of a pressure needs no division (negative_pressure), and a bisection ends when its interval stands still.
// A density wave near vacuum, per launch: P2, 105,456 cells 75 -> 44 us (58 % of issue slots, was 42; 23 million warp
// instructions, were 32) against eight lanes a cell without copies ahead; P1, 131,712 cells 77 -> 48, P3, 48,000 cells
// 87 -> 64.
template <int NB, int NQV>
__global__ void __launch_bounds__(kLimApplyWarps * 32, 2)
    limiter_apply(double* U, const int* __restrict__ nbr, const double* stats, const double* __restrict__ phi, int64_t ncell,
                  double gamma, int only_avg, double* stats_out) {
    using Z = LimSizes<NB, NQV>;
    constexpr int G = Z::G, CPW = Z::CPW, PPL = Z::PPL, GP = Z::GP, B5 = 5 * NB;
    constexpr bool PADS = GP != NQV;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* sphi = reinterpret_cast<double*>(smem_raw);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double* rows = sphi + NB * GP + w * (2 * Z::CHUNK + CPW * 6);
    double* scale = rows + 2 * Z::CHUNK;  // [cell][5 variables, 1 where any is to be stored]
    for (int i = threadIdx.x; i < NB * GP; i += blockDim.x) {
        const int l = i / GP, g = i - l * GP;
        sphi[i] = g < NQV ? phi[g * NB + l] : 0.0;
    }
    __syncthreads();
    const int grp = lane / G, gl = lane - grp * G;
    const int64_t step = (int64_t)gridDim.x * kLimApplyWarps * CPW;
    const bool pairs = (reinterpret_cast<uintptr_t>(U) & 15) == 0;
    auto fetch = [&](int64_t e0, int buf) {
        if (e0 < ncell) {
            const double* from = U + e0 * B5;
            const unsigned to = smem_addr(rows + buf * Z::CHUNK);
            const int len = (int)(ncell - e0 < CPW ? ncell - e0 : CPW) * B5;
            const int even = pairs ? len & ~1 : 0;
            for (int i = 2 * lane; i < even; i += 64)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + 8 * i), "l"(from + i) : "memory");
            for (int i = even + lane; i < len; i += 32)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(to + 8 * i), "l"(from + i) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto cell_of = [&](int64_t e0) { return e0 + grp < ncell ? e0 + grp : ncell - 1; };
    int64_t e0 = ((int64_t)blockIdx.x * kLimApplyWarps + w) * CPW + await_previous();
    int4 n4 = make_int4(0, 0, 0, 0);
    if (e0 < ncell) n4 = __ldg(reinterpret_cast<const int4*>(nbr) + cell_of(e0));
    fetch(e0, 0);
    for (int buf = 0; e0 < ncell; e0 += step, buf ^= 1) {
        const int64_t e = cell_of(e0);
        const bool live = e0 + grp < ncell;
        double* u = rows + buf * Z::CHUNK + (int)(e - e0) * B5;
        // the bounds of neighbour gl (max, min per variable) and this lane's share of the cell's own
        const int64_t nb_cell = (gl & 3) == 0 ? n4.x : (gl & 3) == 1 ? n4.y : (gl & 3) == 2 ? n4.z : n4.w;
        double st[10], own[3];
        #pragma unroll
        for (int i = 0; i < 5; ++i) {
            const double2 x = __ldcg(reinterpret_cast<const double2*>(stats + nb_cell * 10) + i);
            st[2 * i] = x.x;
            st[2 * i + 1] = x.y;
        }
        #pragma unroll
        for (int i = 0; i < 3; ++i) own[i] = __ldcg(stats + e * 10 + min((gl & 3) + 4 * i, 9));
        if (e0 + step < ncell) n4 = __ldg(reinterpret_cast<const int4*>(nbr) + cell_of(e0 + step));
        fetch(e0 + step, buf ^ 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        double v[PPL][5];
        auto evaluate = [&]() {  // summed over the modes in order, as the reference evaluates a point value
            #pragma unroll
            for (int r = 0; r < PPL; ++r)
                #pragma unroll
                for (int k = 0; k < 5; ++k) v[r][k] = 0.0;
            #pragma unroll 2
            for (int l = 0; l < NB; ++l) {
                double c[5];
                #pragma unroll
                for (int k = 0; k < 5; ++k) c[k] = u[5 * l + k];
                #pragma unroll
                for (int r = 0; r < PPL; ++r) {
                    const double p = sphi[l * GP + gl + G * r];
                    #pragma unroll
                    for (int k = 0; k < 5; ++k) v[r][k] = fma(p, c[k], v[r][k]);
                }
            }
        };
        evaluate();
        double avg[5];
        #pragma unroll
        for (int k = 0; k < 5; ++k) avg[k] = u[k];
        if (PADS) {  // neutral in every step
            #pragma unroll
            for (int k = 0; k < 5; ++k)
                if (gl + G * (PPL - 1) >= NQV) v[PPL - 1][k] = avg[k];
        }
        // the cell's bounds: max of maxima, min of last values. A NaN counts only where the cell's own value is
        // one (the comparisons of the reference skip it elsewhere).
        bool own_nan = false;
        #pragma unroll
        for (int i = 0; i < 10; ++i) {
            if (st[i] != st[i]) st[i] = i < 5 ? -DBL_MAX : DBL_MAX;
            const double o = own[i / 4];
            if ((gl & 3) == i % 4) {
                own_nan |= o != o;
                st[i] = i < 5 ? ref_max(st[i], o) : ref_min(st[i], o);
            }
            #pragma unroll
            for (int m = 2; m > 0; m >>= 1) {
                const double other = __shfl_xor_sync(0xffffffffu, st[i], m);
                st[i] = i < 5 ? ref_max(st[i], other) : ref_min(st[i], other);
            }
        }
        if (__any_sync(0xffffffffu, own_nan)) {
            #pragma unroll
            for (int i = 0; i < 10; ++i) {
                const double o = __ldcg(stats + e * 10 + i);
                if (o != o) st[i] = o;
            }
        }
        // step 1: each variable within the cell's bounds. Lane k of a cell forms the quotients of variable k,
        // every lane those of the last one where a cell has four lanes.
        unsigned acts = 0;
        double qa = 0.0, qn = 0.0, qx = 0.0, qb = 0.0, qm = 0.0, last = 1.0;
        double vmax[5];
        #pragma unroll
        for (int k = 0; k < 5; ++k) {
            double mn = DBL_MAX, mx = -DBL_MAX;
            #pragma unroll
            for (int r = 0; r < PPL; ++r)
                if (gl + G * r < NQV) { mn = ref_min(mn, v[r][k]); mx = ref_max(mx, v[r][k]); }
            mn = group_min<G>(mn, 0xffffffffu);
            mx = group_max<G>(mx, 0xffffffffu);
            vmax[k] = mx;
            bool out = mn < st[5 + k] || mx > st[k];
            if (PADS) out |= avg[k] < st[5 + k] || avg[k] > st[k];
            if (out) acts |= 1u << k;
            if (G > 4 || k < 4) {
                if (gl == k) { qa = avg[k]; qn = mn; qx = mx; qb = st[5 + k]; qm = st[k]; }
            } else {
                last = limiter_theta(avg[k], mn, mx, st[5 + k], st[k]);
            }
        }
        double s[5] = {1.0, 1.0, 1.0, 1.0, 1.0};  // per-variable scale of modes l >= 1
        if (__any_sync(0xffffffffu, acts != 0u)) {
            const double mine = limiter_theta(qa, qn, qx, qb, qm);
            #pragma unroll
            for (int k = 0; k < 5; ++k) {
                const double theta = G > 4 || k < 4 ? __shfl_sync(0xffffffffu, mine, k, G) : last;
                if (acts >> k & 1u) {
                    s[k] = theta;
                    #pragma unroll
                    for (int r = 0; r < PPL; ++r) v[r][k] = avg[k] + theta * (v[r][k] - avg[k]);
                }
            }
        }
        // step 2: density at the points >= 1e-16
        {
            const double eps = 1e-16;
            double rmin = DBL_MAX;
            bool low = false;
            #pragma unroll
            for (int r = 0; r < PPL; ++r) {
                low |= v[r][0] < eps;
                if (gl + G * r < NQV) rmin = ref_min(rmin, v[r][0]);
            }
            if (__any_sync(0xffffffffu, low)) {
                rmin = group_min<G>(rmin, 0xffffffffu);
                if (__ballot_sync(0xffffffffu, low) >> (lane - gl) & ((1ull << G) - 1)) {
                    const double eff = ref_max(avg[0], eps);
                    const double num = eff - eps, den = eff - rmin;
                    const double theta = (den < 1e-32) ? 0.0 : ref_min(1.0, num / den);
                    s[0] *= theta;
                    #pragma unroll
                    for (int r = 0; r < PPL; ++r) v[r][0] = avg[0] + theta * (v[r][0] - avg[0]);
                    acts |= 1u;
                }
            }
        }
        // step 3: pressure at the points >= 0 by bisection toward the mean
        double tp = 1.0;
        unsigned neg = 0;
        #pragma unroll
        for (int r = 0; r < PPL; ++r)
            if (gl + G * r < NQV && negative_pressure(v[r], gamma)) neg |= 1u << r;
        if (__any_sync(0xffffffffu, neg != 0u)) {
            #pragma unroll
            for (int r = 0; r < PPL; ++r) {
                if (!(neg >> r & 1u)) continue;
                double lo = 0.0, hi = 1.0, mid = 0.5 * (lo + hi);
                for (int it = 0; it < 100; ++it) {
                    mid = 0.5 * (lo + hi);
                    double um[5];
                    #pragma unroll
                    for (int k = 0; k < 5; ++k) um[k] = (1.0 - mid) * avg[k] + mid * v[r][k];
                    const bool low_side = negative_pressure(um, gamma);
                    if (mid == (low_side ? hi : lo)) break;  // every further step would be the same
                    if (low_side) hi = mid;
                    else lo = mid;
                }
                tp = ref_min(tp, mid);
            }
            __syncwarp();
            tp = group_min<G>(tp, 0xffffffffu);
        }
        const bool changed = acts != 0u || tp != 1.0;
        if (__any_sync(0xffffffffu, changed)) {  // modes l >= 1: c *= theta_1 [*= theta_rho] *= theta_p, in the reference's order
            if (gl == 0) {
                #pragma unroll
                for (int k = 0; k < 5; ++k) scale[grp * 6 + k] = s[k];
            }
            __syncwarp();
            double* chunk = rows + buf * Z::CHUNK;
            for (int i0 = 0; i0 < Z::CHUNK; i0 += 32) {
                const int i = i0 + lane, c = min(i / B5, CPW - 1), rr = i - c * B5;
                // the pressure scale and the flag are the cell's lanes': taken by shuffle
                const double t = __shfl_sync(0xffffffffu, tp, c * G);
                const bool act = __shfl_sync(0xffffffffu, (int)(changed && live), c * G);
                if (act && i < Z::CHUNK && rr >= 5) {
                    const double x = chunk[i] * scale[c * 6 + rr % 5] * t;
                    chunk[i] = x;
                    U[e0 * B5 + i] = x;
                }
            }
            __syncwarp();
            if (stats_out && !only_avg) {  // the limited state's point values, re-evaluated
                evaluate();
                write_stats<NQV, G, PPL>(v, avg, gl, 0xffffffffu, 0, stats_out + e * 10, live);
            }
        } else if (stats_out && !only_avg && live) {
            constexpr int LR = (NQV - 1) / G, LL = (NQV - 1) % G;
            #pragma unroll
            for (int k = 0; k < 5; ++k) {
                if (gl == LL) stats_out[e * 10 + 5 + k] = v[LR][k];
                if (gl == 0) stats_out[e * 10 + k] = vmax[k];
            }
        }
        if (stats_out && only_avg) write_stats<NQV, G, PPL>(v, avg, gl, 0xffffffffu, 1, stats_out + e * 10, live);
        __syncwarp();  // the buffer is free
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    release_next();
}

// X(order, qv, NB, NQV)
#define FVEDG_LIMITER_COMBOS(X) \
    X(1, 0, 4, 4)               \
    X(1, 2, 4, 15)              \
    X(2, 1, 10, 11)             \
    X(2, 2, 10, 15)             \
    X(3, 3, 20, 23)             \
    X(3, 4, 20, 31)             \
    X(4, 5, 35, 44)             \
    X(4, 6, 35, 57)

template <int NB, int NQV>
inline int run_limiter_apply(double* U, const int* nbr, const double* stats, const double* phi, int64_t ncell, double gamma,
                             int only_avg, double* stats_out, int sms, cudaStream_t s) {
    using Z = LimSizes<NB, NQV>;
    static unsigned long long done = 0;
    if (const int rc = ensure_smem(limiter_apply<NB, NQV>, Z::smem, done)) return rc;
    const int64_t per_block = kLimApplyWarps * Z::CPW;
    const int g = (int)std::max<int64_t>(1, std::min<int64_t>((ncell + per_block - 1) / per_block, 2 * (int64_t)sms));
    return launch_early(limiter_apply<NB, NQV>, g, kLimApplyWarps * 32, Z::smem, s, U, nbr, stats, phi, ncell, gamma, only_avg,
                        stats_out);
}

inline bool limiter_supported(int order, int qv) {
#define X(P, QV, NB, NQV) \
    if (order == P && qv == QV) return true;
    FVEDG_LIMITER_COMBOS(X)
#undef X
    return false;
}

// Bounds from Uprev, then the three steps on U (in place) for cells [0, napply) (the owned cells;
// the statistics cover ghost cells too). stats: [ncell][10] scratch.
inline int launch_limiter(int order, int qv, double* U, const double* Uprev, const int* nbr, const double* phi_v,
                          int64_t ncell, int64_t napply, double gamma, int only_avg, double* stats, int sms,
                          cudaStream_t s) {
#define X(P, QV, NB, NQV)                                                                                        \
    if (order == P && qv == QV) {                                                                                \
        const unsigned ge = (unsigned)std::min<int64_t>((ncell + kLimWarps - 1) / kLimWarps, (int64_t)sms * 16); \
        limiter_cell_stats<NB, NQV><<<ge, kLimWarps * 32, 0, s>>>(Uprev, phi_v, 0, ncell, only_avg, stats);      \
        const int rc = cuda_status(cudaGetLastError());                                                          \
        if (rc) return rc;                                                                                       \
        return run_limiter_apply<NB, NQV>(U, nbr, stats, phi_v, napply, gamma, only_avg, nullptr, sms, s);       \
    }
    FVEDG_LIMITER_COMBOS(X)
#undef X
    return DG_E_ARG;
}

// Statistics of cells [c_begin, c_end) of U into stats.
inline int launch_limiter_stats(int order, int qv, const double* U, const double* phi_v, int64_t c_begin,
                                int64_t c_end, int only_avg, double* stats, int sms, cudaStream_t s,
                                std::atomic<int64_t>* launches) {
    if (c_begin >= c_end) return DG_OK;
#define X(P, QV, NB, NQV)                                                                                       \
    if (order == P && qv == QV) {                                                                               \
        const int64_t n = c_end - c_begin;                                                                      \
        const unsigned gs = (unsigned)std::min<int64_t>((n + kLimWarps - 1) / kLimWarps, (int64_t)sms * 16);    \
        limiter_cell_stats<NB, NQV><<<gs, kLimWarps * 32, 0, s>>>(U, phi_v, c_begin, c_end, only_avg, stats);   \
        ++*launches;                                                                                            \
        return cuda_status(cudaGetLastError());                                           \
    }
    FVEDG_LIMITER_COMBOS(X)
#undef X
    return DG_E_ARG;
}

// The limiter inside the time loop, one launch per stage: bounds from `stats_in` (the statistics
// of the stage input, which the previous stage's launch wrote), and the statistics of the limited
// output into `stats_out`. The statistics of cells [stats_begin, ncell) of the input are computed
// first (all cells after the state was set from outside, else the ghost cells, whose rows a halo
// exchange rewrote; none when stats_begin == ncell).
inline int launch_limiter_stage(int order, int qv, double* U, const double* Uin, const int* nbr, const double* phi_v,
                                int64_t ncell, int64_t napply, int64_t stats_begin, double gamma, int only_avg,
                                double* stats_in, double* stats_out, int sms, cudaStream_t s,
                                std::atomic<int64_t>* launches) {
    int rc = launch_limiter_stats(order, qv, Uin, phi_v, stats_begin, ncell, only_avg, stats_in, sms, s, launches);
    if (rc) return rc;
#define X(P, QV, NB, NQV)                                                                                         \
    if (order == P && qv == QV) {                                                                                 \
        ++*launches;                                                                                              \
        return run_limiter_apply<NB, NQV>(U, nbr, stats_in, phi_v, napply, gamma, only_avg, stats_out, sms, s);   \
    }
    FVEDG_LIMITER_COMBOS(X)
#undef X
    return DG_E_ARG;
}

}  // namespace fvedg
