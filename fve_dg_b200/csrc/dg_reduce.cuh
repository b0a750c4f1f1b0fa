// Deterministic reductions over the device state: conservation sums, the largest wave speed (for a
// CFL time step, cf. examples/TaylerGreenVortex/TGBatch.cpp:358-383) and the non-physical point
// count. One launch of partial sums per block (a fixed assignment of elements to warps and of points
// to lanes) and one that adds them in a fixed order, so results do not depend on scheduling.
#pragma once
#include <algorithm>
#include <atomic>
#include <cstdint>

#include "dg_flux.cuh"
#include "dg_kernels_fp64_rows.cuh"
#include "dg_launch.cuh"
#include "dg_mixed_host.cuh"

namespace fvedg {

constexpr int kRedMaxBlocks = 592;  // 4 x 148 SMs: what the partials have room for
constexpr int kRedMaxWarps = 16;

enum RedKind { RED_CONSERVATION = 0, RED_WAVESPEED = 1, RED_BADPOINTS = 2 };

template <int KIND>
__device__ __forceinline__ double red_combine(double a, double b) {
    return KIND == RED_WAVESPEED ? fmax(a, b) : a + b;
}

// Shared memory of the partial sums: the volume basis as B operands [point tile][k-tile][lane], the weights, and per
// warp two buffers of eight elements' rows.
struct RedSizes {
    int nt, kt, warps;
    size_t table, chunk;
    RedSizes(int nb, int nqv)
        : nt((nqv + 7) / 8), kt((nb + 3) / 4), table(((size_t)nt * kt * 32 + (nqv + 1) / 2 * 2) * 8), chunk((size_t)8 * 5 * nb * 8) {
        warps = (int)std::min<size_t>(kRedMaxWarps, (220 * 1024 - table) / (2 * chunk));
    }
    size_t smem() const { return table + 2 * chunk * warps; }
};

// partial[block][0..5]. A warp takes eight consecutive elements, whose rows are one piece of memory, and evaluates
// their point values on the FP64 tensor cores as the element kernels do: item = row, variable = tile, the five values
// of a point in one lane's accumulators. The next rows are on their way meanwhile. Bound by the FP64 pipe (P3: 75
// tensor instructions and six points a lane, with a division and two square roots each for the wave speed, per
// eight elements). The wave speed of 279,936 P3 elements, with its sum and the host's read: 460 us with one element per
// warp and scalar sums read from global memory, of which the last block's serial pass was a part; 150 here.
template <int KIND>
__global__ void __launch_bounds__(kRedMaxWarps * 32, 1) state_reduce_kernel(const double* U, const double* __restrict__ geo,
        const double* __restrict__ phi_v, const double* __restrict__ w_v, int ncell, int nb, int nqv, int ntile, int ktile,
        double gamma, double* partial) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double sh[kRedMaxWarps][6];
    double* tab = reinterpret_cast<double*>(smem_raw);
    double* w = tab + ntile * ktile * 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tq = lane & 3;
    const int nw = blockDim.x >> 5, b5 = 5 * nb;
    double* rows = w + (nqv + 1) / 2 * 2 + warp * 2 * 8 * b5;
    for (int i = threadIdx.x; i < ntile * ktile * 32; i += blockDim.x) {
        const int l = i & 31, t = i >> 5, g = 8 * (t / ktile) + (l >> 2), b = 4 * (t % ktile) + (l & 3);
        tab[i] = g < nqv && b < nb ? phi_v[g * nb + b] : 0.0;
    }
    if (KIND == RED_CONSERVATION)
        for (int i = threadIdx.x; i < nqv; i += blockDim.x) w[i] = w_v[i];
    __syncthreads();
    const int ngroups = (ncell + 7) / 8, step = gridDim.x * nw;
    auto fetch = [&](int gi, int buf) {  // the group's rows, in copies of two doubles and an odd last one
        if (gi < ngroups) {
            const double* from = U + (int64_t)gi * 8 * b5;
            const unsigned to = smem_addr(rows + buf * 8 * b5);
            const int len = min(8, ncell - 8 * gi) * b5;
            for (int i = 2 * lane; i + 1 < len; i += 64)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + 8 * i), "l"(from + i) : "memory");
            if ((len & 1) && lane == 0)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(to + 8 * (len - 1)), "l"(from + len - 1) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    double acc[6] = {0, 0, 0, 0, 0, 0};
    int gi = blockIdx.x + gridDim.x * warp + await_previous(), buf = 0;
    fetch(gi, 0);
    for (; gi < ngroups; gi += step, buf ^= 1) {
        fetch(gi + step, buf ^ 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        const int64_t e = (int64_t)gi * 8 + gid;
        const bool live = e < ncell;
        const double* row = rows + (buf * 8 + gid) * b5;
        const double dj = KIND == RED_CONSERVATION && live ? geo[e * 10 + 9] : 0.0;
        if (KIND == RED_CONSERVATION && live && tq == 0)
            for (int k = 0; k < 5; ++k) acc[k] += row[k] * dj / 6.0;
        for (int nt = 0; nt < ntile; ++nt) {
            double v[5][2];
            #pragma unroll
            for (int k = 0; k < 5; ++k) v[k][0] = v[k][1] = 0.0;
            const double* tb = tab + nt * ktile * 32 + lane;
            #pragma unroll 2
            for (int kt = 0; kt < ktile; ++kt) {
                const int b = 4 * kt + tq;
                const double t = tb[kt * 32];
                #pragma unroll
                for (int k = 0; k < 5; ++k) dmma884(v[k], b < nb ? row[5 * b + k] : 0.0, t);
            }
            #pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int g = 8 * nt + 2 * tq + i;
                if (!live || g >= nqv) continue;
                const double m2 = v[1][i] * v[1][i] + v[2][i] * v[2][i] + v[3][i] * v[3][i];
                if (KIND == RED_CONSERVATION) {
                    acc[5] += w[g] * dj * 0.5 * m2 / Phys<double>::positive(v[0][i]);
                } else {
                    const double rho = v[0][i], ir = 1.0 / rho;
                    const double p = (gamma - 1.0) * (v[4][i] - 0.5 * m2 * ir);
                    bool bad = !(rho > 0.0) || !(p > 0.0);
                    #pragma unroll
                    for (int k = 0; k < 5; ++k) bad = bad || !isfinite(v[k][i]);
                    if (KIND == RED_BADPOINTS) {
                        acc[0] += bad ? 1.0 : 0.0;
                    } else if (!bad) {
                        const double u0 = v[1][i] * ir, u1 = v[2][i] * ir, u2 = v[3][i] * ir;
                        acc[0] = fmax(acc[0], sqrt(u0 * u0 + u1 * u1 + u2 * u2) + sqrt(gamma * Phys<double>::positive(p * ir)));
                    }
                }
            }
        }
        __syncwarp();  // the buffer is free
    }
    release_next();
    #pragma unroll
    for (int k = 0; k < 6; ++k) {
        #pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[k] = red_combine<KIND>(acc[k], __shfl_down_sync(0xffffffffu, acc[k], o));
        if (lane == 0) sh[warp][k] = acc[k];
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        double s = sh[0][threadIdx.x];
        for (int i = 1; i < nw; ++i) s = red_combine<KIND>(s, sh[i][threadIdx.x]);
        partial[blockIdx.x * 6 + threadIdx.x] = s;
    }
}

// Warp k adds component k of the blocks' partial sums.
template <int KIND>
__global__ void __launch_bounds__(192) partial_sum_kernel(const double* partial, int nblk, double* out) {
    const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double s = 0.0;
    for (int b = lane + await_previous(); b < nblk; b += 32) s = red_combine<KIND>(s, __ldcg(partial + b * 6 + k));
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) s = red_combine<KIND>(s, __shfl_down_sync(0xffffffffu, s, o));
    if (lane == 0) out[k] = s;
}

template <int KIND>
inline int run_state_reduce(const double* U, const double* geo, const double* phi_v, const double* w_v, int ncell,
                            int nb, int nqv, double gamma, int sms, double* partial, double out[6],
                            cudaStream_t s, std::atomic<int64_t>* launches) {
    const RedSizes z(nb, nqv);
    static unsigned long long done = 0;
    if (const int rc = ensure_smem(state_reduce_kernel<KIND>, 226 * 1024, done)) return rc;
    const int blocks = std::max(1, std::min({sms, kRedMaxBlocks, (ncell + 7) / 8}));
    int rc = launch_early(state_reduce_kernel<KIND>, blocks, z.warps * 32, z.smem(), s, U, geo, phi_v, w_v, ncell, nb, nqv,
                          z.nt, z.kt, gamma, partial);
    if (rc == DG_OK) rc = launch_early(partial_sum_kernel<KIND>, 1, 192, 0, s, partial, blocks, partial + (size_t)kRedMaxBlocks * 6);
    *launches += 2;
    if (rc) return rc;
    if ((rc = cuda_status(cudaMemcpyAsync(out, partial + (size_t)kRedMaxBlocks * 6, 6 * sizeof(double), cudaMemcpyDeviceToHost, s))))
        return rc;
    return cuda_status(cudaStreamSynchronize(s));
}

inline int reduce_conservation(const double* U, const double* geo, const double* phi_v, const double* w_v,
                               int ncell, int nb, int nqv, int sms, double* partial, double out[6], cudaStream_t s,
                               std::atomic<int64_t>* launches) {
    return run_state_reduce<RED_CONSERVATION>(U, geo, phi_v, w_v, ncell, nb, nqv, 1.4, sms, partial, out, s, launches);
}
inline int reduce_wave_speed(const double* U, const double* phi_v, int ncell, int nb, int nqv, double gamma, int sms,
                             double* partial, double* lam, cudaStream_t s, std::atomic<int64_t>* launches) {
    double o[6];
    int rc = run_state_reduce<RED_WAVESPEED>(U, nullptr, phi_v, nullptr, ncell, nb, nqv, gamma, sms, partial, o, s, launches);
    *lam = o[0];
    return rc;
}
inline int reduce_bad_points(const double* U, const double* phi_v, int ncell, int nb, int nqv, double gamma, int sms,
                             double* partial, double* nbad, cudaStream_t s, std::atomic<int64_t>* launches) {
    double o[6];
    int rc = run_state_reduce<RED_BADPOINTS>(U, nullptr, phi_v, nullptr, ncell, nb, nqv, gamma, sms, partial, o, s, launches);
    *nbad = o[0];
    return rc;
}

}  // namespace fvedg
