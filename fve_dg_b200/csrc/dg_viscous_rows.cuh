// The explicit viscous operator (dg_viscous.cuh has its terms and their origin) in rows of eight items, FP64: the
// layout of dg_kernels_fp64_rows.cuh, where a lane's accumulators hold all five variables, and here their three
// reference derivatives too, of one item at the same two points. Nothing but the state rows passes through
// shared memory.
//
//   face      values and reference gradients of both sides (20 products per k-tile and side on one set of A
//             operands), the averaged flux with its penalty folded into the gradient (X - beta dU n, one
//             contraction), its moments; the symmetric term's source s as a sixth column of moments S_m, and
//             from them T_j = sum_m S_m (n_L . D^L_jm + n_R . D^R_jm) with D[perm][d][j][m] the moments of the
//             reference derivative of mode j (a polynomial on the face like any other)
//   element   values and gradients, the flux pulled back to reference directions, its volume integral, the four
//             faces' moments with T[perm] and T_j in the energy column
//
// The mass equation has no viscous flux: its tile is left out of every integral.
//
// Fused: with CONV the same launches add the convective terms (the Navier-Stokes stage R_conv - R_visc): the traces,
// the volume values and the face integrals are then formed once for both, and no viscous residual is stored.
//
// Bound: the FP64 pipe, which the tensor instruction and DFMA share. Fused P3 launches at 82,944 cells: faces 415 us,
// elements 212 us, the tensor instruction alone 48 % and 50 % of the pipe's cycles, DRAM 3 % and 14 % (the state and the
// records stay in L2). A Navier-Stokes step: 5,800 us with one warp per item and four launches a stage (two of them
// with point values in shared memory and scalar contractions), 5,627 with only the convective launches in rows of eight,
// 2,053 fused. Eight warps per SM, for the 255 registers that the values and three gradients of five variables need.
#pragma once
#include "dg_kernels_fp64_rows.cuh"
#include "dg_viscous.cuh"

namespace fvedg {

struct Visc8Tables {
    const double* tfd;  // [24][point tile][k-tile][direction][lane]  dphi_f: mode 4 kt + tq at point 8 nt + gid
    const double* tvd;  // [point tile][k-tile][direction][lane]  dphi_v
    const double* td;   // [24][direction][k-tile][mode tile][lane]  D[perm]: moment 8 (kt / 2) + 2 tq + kt % 2, mode 8 j + gid
};

// Moments of the derivatives (degree P - 1) come in the first k-tiles; the record's doubles.
__host__ __device__ constexpr int deriv_ktiles(int nb) { return nb <= 20 ? 2 : 4; }
__host__ __device__ constexpr int visc_rec(int nb) { return 5 * moment_row(nb) + (nb + 1) / 2 * 2; }

struct Visc8Args {
    Rows8FaceArgs f;     // U, faces, groups, UD, tables; rec is [nface][visc_rec]
    Rows8ElemArgs e;     // elements; mode 0: out = R_visc, mode 1 (CONV): the stage update with R_conv - R_visc
    Visc8Tables v;
    const double* geo;   // [ncell][10]: J^-T row-major, detJ
    const double* h;     // [ncell] volume / sum of face areas
    double mu, cq;       // viscosity and gamma / Pr
    int order;
};

// Values and reference gradients at the points 8 nt + 2 tq + {0, 1} of the lane's row.
template <int NB>
__device__ __forceinline__ void gradients8(double (&v)[5][2], double (&g)[3][5][2], const double* row,
                                           const double* __restrict__ tv, const double* __restrict__ td, int lane) {
    constexpr int KT = (NB + 3) / 4;
    const int tq = lane & 3;
    #pragma unroll
    for (int k = 0; k < 5; ++k) {
        v[k][0] = v[k][1] = 0.0;
        #pragma unroll
        for (int d = 0; d < 3; ++d) g[d][k][0] = g[d][k][1] = 0.0;
    }
    #pragma unroll
    for (int kt = 0; kt < KT; ++kt) {
        const double b = __ldg(tv + kt * 32 + lane);
        double bd[3], c[5];
        #pragma unroll
        for (int d = 0; d < 3; ++d) bd[d] = __ldg(td + (kt * 3 + d) * 32 + lane);
        const bool on = 4 * kt + 3 < NB || 4 * kt + tq < NB;
        #pragma unroll
        for (int k = 0; k < 5; ++k) c[k] = on ? row[5 * (4 * kt + tq) + k] : 0.0;
        #pragma unroll
        for (int k = 0; k < 5; ++k) dmma884(v[k], c[k], b);
        #pragma unroll
        for (int d = 0; d < 3; ++d)
            #pragma unroll
            for (int k = 0; k < 5; ++k) dmma884(g[d][k], c[k], bd[d]);
    }
}

// sum_n n_n H_n[i], i = 1..4, for gradients X[k][m] at the state s (visc_contract of dg_viscous.cuh along one
// direction): Y_a,m = (X_a+1,m - u_a X_0,m) / rho, F_a = mu (Y_a. n + n_a tr Y - 2/3 n . Y_.a).
__device__ __forceinline__ void visc_flux_n(const ViscState& s, double mu, double cq, const double (&X)[5][3],
                                            const double n[3], double F[5]) {
    double Xn[5];
    #pragma unroll
    for (int k = 0; k < 5; ++k) Xn[k] = X[k][0] * n[0] + X[k][1] * n[1] + X[k][2] * n[2];
    const double un = s.u[0] * n[0] + s.u[1] * n[1] + s.u[2] * n[2];
    double tr = 0.0, yn[3];
    #pragma unroll
    for (int a = 0; a < 3; ++a) {
        tr += X[1 + a][a] - s.u[a] * X[0][a];
        yn[a] = Xn[1 + a] - s.u[a] * Xn[0];
    }
    const double m = mu * s.irho;
    F[0] = 0.0;
    #pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double yt = n[0] * X[1][a] + n[1] * X[2][a] + n[2] * X[3][a] - un * X[0][a];
        F[1 + a] = m * (yn[a] + n[a] * tr - (2.0 / 3.0) * yt);
    }
    const double ye = Xn[4] - s.e * Xn[0] - (s.u[0] * yn[0] + s.u[1] * yn[1] + s.u[2] * yn[2]);
    F[4] = s.u[0] * F[1] + s.u[1] * F[2] + s.u[2] * F[3] + m * cq * ye;
}

// H[n][i], i = 1..4, for all three directions.
__device__ __forceinline__ void visc_flux_3(const ViscState& s, double mu, double cq, const double (&X)[5][3], double (&H)[3][5]) {
    double Y[3][3], tr = 0.0;
    #pragma unroll
    for (int a = 0; a < 3; ++a) {
        #pragma unroll
        for (int m = 0; m < 3; ++m) Y[a][m] = X[1 + a][m] - s.u[a] * X[0][m];
        tr += Y[a][a];
    }
    const double m = mu * s.irho;
    #pragma unroll
    for (int n = 0; n < 3; ++n) {
        H[n][0] = 0.0;
        #pragma unroll
        for (int a = 0; a < 3; ++a) H[n][1 + a] = m * (Y[a][n] + (a == n ? tr : 0.0) - (2.0 / 3.0) * Y[n][a]);
        const double ye = X[4][n] - s.e * X[0][n] - (s.u[0] * Y[0][n] + s.u[1] * Y[1][n] + s.u[2] * Y[2][n]);
        H[n][4] = s.u[0] * H[n][1] + s.u[1] * H[n][2] + s.u[2] * H[n][3] + m * cq * ye;
    }
}

template <int NB, int NQF, bool CONV>
__device__ __forceinline__ bool visc_face_group8(const Visc8Args& A, int gi, FaceSmem8<NB>& sm, uint64_t& bar,
                                                 unsigned& parity, int lane) {
    using Slots = Slots8<NB>;
    const Rows8FaceArgs& a = A.f;
    constexpr int B5 = 5 * NB, NT = pad8(NQF) / 8, KT = (NB + 3) / 4, NJ = pad8(NB) / 8, MR = moment_row(NB), MT = (MR + 7) / 8;
    constexpr int RW = visc_rec(NB), KD = deriv_ktiles(NB), K0 = CONV ? 0 : 1;
    const int gid = lane >> 2, tq = lane & 3;
    const FaceGroup8& grp = a.groups[gi];
    const int n = grp.n, f = grp.f[gid];
    const FaceInfo F = a.fi[f];
    if (!visc_face_active(F, a.UD)) {  // shared by the group
        for (int i = lane; i < n * RW; i += 32) a.rec[(int64_t)grp.f[i / RW] * RW + i % RW] = 0.0;
        return true;
    }
    const int bc = (F.meta >> 16) & 0xff;
    const bool interior = F.c1 >= 0;
    {   // lane i < 16 moves the row of cells[i / 8] of face i % 8 (a boundary face's one cell twice)
        const FaceInfo& mine = a.fi[grp.f[lane & 7]];
        const int c = (lane & 8) && interior ? mine.c1 : mine.c0;
        Slots::load(sm.rows, lane, 16, a.U + (int64_t)c * B5, &bar);
    }
    const double beta = (double)((A.order + 1) * (A.order + 1)) / A.h[F.c0], half = interior ? 0.5 : 1.0;
    const int nside = interior ? 2 : 1;
    double mom[6][MT][2];  // moments of the flux, then of s
    #pragma unroll
    for (int k = 0; k < 6; ++k)
        #pragma unroll
        for (int mt = 0; mt < MT; ++mt) mom[k][mt][0] = mom[k][mt][1] = 0.0;
    if (!rows_landed<true>(bar, parity, a.err)) return false;
    #pragma unroll 1
    for (int nt = 0; nt < NT; ++nt) {
        double V[2][5][2], X[2][5][3];  // [point]: averaged (boundary: inner) physical gradient
        #pragma unroll
        for (int i = 0; i < 2; ++i)
            #pragma unroll
            for (int k = 0; k < 5; ++k) X[i][k][0] = X[i][k][1] = X[i][k][2] = 0.0;
        #pragma unroll
        for (int s = 0; s < 2; ++s) {
            if (s >= nside) continue;
            const int cell = s ? F.c1 : F.c0, perm = (F.meta >> (8 * s)) & 0xff;
            double G[3][5][2];
            gradients8<NB>(V[s], G, Slots::at(sm.rows, gid + 8 * s, a.U + (int64_t)cell * B5),
                           a.t.tf + (int64_t)(perm * NT + nt) * KT * 32, A.v.tfd + (int64_t)(perm * NT + nt) * KT * 96, lane);
            #pragma unroll
            for (int m = 0; m < 3; ++m)
                #pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const double J = half * __ldg(A.geo + (int64_t)cell * 10 + 3 * m + d);
                    #pragma unroll
                    for (int k = 0; k < 5; ++k)
                        #pragma unroll
                        for (int i = 0; i < 2; ++i) X[i][k][m] = fma(J, G[d][k][i], X[i][k][m]);
                }
        }
        double O[6][2];  // what the moments are taken of
        #pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int g = nt * 8 + 2 * tq + i;
            const bool pad = NQF % 8 != 0 && g >= NQF;
            double UL[5], UR[5], Um[5], Fv[5];
            #pragma unroll
            for (int k = 0; k < 5; ++k) UL[k] = V[0][k][i];
            if (interior) {
                #pragma unroll
                for (int k = 0; k < 5; ++k) UR[k] = V[1][k][i];
            } else if (bc == 0) {
                const double* ud = a.UD + ((int64_t)f * NQF + (pad ? 0 : g)) * 5;
                #pragma unroll
                for (int k = 0; k < 5; ++k) UR[k] = ud[k] + (ud[k] - UL[k]);  // ghost 2 U_D - U
            } else {
                #pragma unroll
                for (int k = 0; k < 5; ++k) UR[k] = UL[k];
                UR[3] = -UL[3];
            }
            #pragma unroll
            for (int k = 0; k < 5; ++k) {
                Um[k] = 0.5 * (UL[k] + UR[k]);
                const double dU = beta * (interior ? UL[k] - UR[k] : UL[k]);
                #pragma unroll
                for (int m = 0; m < 3; ++m) X[i][k][m] = fma(-dU, F.n[m], X[i][k][m]);
            }
            const ViscState st = visc_state(Um);
            visc_flux_n(st, A.mu, A.cq, X[i], F.n, Fv);
            const double s = half * A.mu * A.cq * st.irho * (UR[4] - UL[4]);
            if (CONV) {
                double Fc[5];
                if (a.flux == 1) roe_f64(UL, UR, F.n, a.gamma, Fc);
                else lax_friedrichs_f64(UL, UR, F.n, a.gamma, Fc);
                #pragma unroll
                for (int k = 0; k < 5; ++k) Fv[k] = Fc[k] - Fv[k];
            }
            #pragma unroll
            for (int k = K0; k < 5; ++k) O[k][i] = pad ? 0.0 : Fv[k];
            O[5][i] = pad ? 0.0 : (CONV ? -s : s);
        }
        #pragma unroll
        for (int i = 0; i < 2; ++i)
            #pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
                const double b = __ldg(a.t.tm + ((nt * 2 + i) * MT + mt) * 32 + lane);
                #pragma unroll
                for (int k = K0; k < 6; ++k) dmma884(mom[k][mt], O[k][i], b);
            }
    }
    __syncwarp();  // the slots are free
    // T_j per mode, the same for both sides up to sign
    double T[NJ][2];
    #pragma unroll
    for (int j = 0; j < NJ; ++j) T[j][0] = T[j][1] = 0.0;
    for (int s = 0; s < nside; ++s) {
        const double* J = A.geo + (int64_t)(s ? F.c1 : F.c0) * 10;
        const double* td = A.v.td + (int64_t)((F.meta >> (8 * s)) & 0xff) * 3 * KD * NJ * 32 + lane;
        #pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double nd = F.jw * (__ldg(J + d) * F.n[0] + __ldg(J + 3 + d) * F.n[1] + __ldg(J + 6 + d) * F.n[2]);
            #pragma unroll
            for (int t = 0; t < KD; ++t) {
                const double x = nd * mom[5][t / 2][t % 2];
                #pragma unroll
                for (int j = 0; j < NJ; ++j) dmma884(T[j], x, __ldg(td + ((d * KD + t) * NJ + j) * 32));
            }
        }
    }
    if (gid < n) {
        double* rec = a.rec + (int64_t)f * RW;
        #pragma unroll
        for (int mt = 0; mt < MT; ++mt)
            if (8 * mt + 2 * tq < MR)
                #pragma unroll
                for (int k = K0; k < 5; ++k)
                    *reinterpret_cast<double2*>(rec + k * MR + 8 * mt + 2 * tq) = make_double2(mom[k][mt][0] * F.jw, mom[k][mt][1] * F.jw);
        #pragma unroll
        for (int j = 0; j < NJ; ++j)
            if (8 * j + 2 * tq < NB) *reinterpret_cast<double2*>(rec + 5 * MR + 8 * j + 2 * tq) = make_double2(T[j][0], T[j][1]);
    }
    return true;
}

template <int NB, int NQF, bool CONV, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 1) visc_face_rows8(Visc8Args A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint64_t bars[WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto& sm = reinterpret_cast<FaceSmem8<NB>*>(smem_raw)[warp];
    if (lane == 0) mbar_init(&bars[warp], 16);
    __syncwarp();
    unsigned parity = 0;
    for (int gi = blockIdx.x + gridDim.x * warp + await_previous(); gi < A.f.ngroups; gi += gridDim.x * WARPS) {
        if (gi + gridDim.x * WARPS >= A.f.ngroups) release_next();
        if (!visc_face_group8<NB, NQF, CONV>(A, gi, sm, bars[warp], parity, lane)) break;
    }
}

template <int NB, int NQV, bool CONV>
__device__ __forceinline__ bool visc_element_group8(const Visc8Args& A, int gi, ElemSmem8<NB>& sm, uint64_t& bar,
                                                    unsigned& parity, int lane) {
    using Slots = Slots8<NB>;
    const Rows8ElemArgs& a = A.e;
    constexpr int B5 = 5 * NB, NT = pad8(NQV) / 8, KT = (NB + 3) / 4, NJ = pad8(NB) / 8, MR = moment_row(NB);
    constexpr int KF = moment_ktiles(NB), RW = visc_rec(NB), K0 = CONV ? 0 : 1;
    const int gid = lane >> 2, tq = lane & 3;
    if (lane < (int)(sizeof(ElemGroup8) / 16))
        reinterpret_cast<uint4*>(&sm.grp)[lane] = __ldg(reinterpret_cast<const uint4*>(a.groups + gi) + lane);
    __syncwarp();
    const ElemGroup8& grp = sm.grp;
    const int n = grp.n;
    const int64_t e = grp.e[gid];
    const bool u0 = CONV && a.mode != 0 && a.a0 != 0.0;
    {   // lane i < 8: the stage input's row i; lane 8 + i: U^n's
        const int64_t mine = grp.e[lane & 7];
        Slots::load(sm.rows, lane, 8, a.U + mine * B5, &bar);
        if (lane >= 8 && lane < 16) {
            if (u0) Slots::load(sm.rows0, lane - 8, 8, a.U0 + mine * B5, &bar);
            else mbar_arrive(&bar);
        }
    }
    {   // the face records into L2 while the volume term is computed
        constexpr int NL = (RW * 8 + 127) / 128;
        for (int i = lane; i < 4 * kRows8 * NL; i += 32) {
            const int fq = i / NL, part = i - fq * NL;
            prefetch_l2(reinterpret_cast<const char*>(a.rec + (int64_t)grp.face[fq >> 2][fq & 3] * RW) + min(part * 128, RW * 8 - 8));
        }
    }
    double J[9];
    const double detj = __ldg(A.geo + e * 10 + 9);
    #pragma unroll
    for (int i = 0; i < 9; ++i) J[i] = __ldg(A.geo + e * 10 + i);
    double acc[5][NJ][2];
    #pragma unroll
    for (int k = 0; k < 5; ++k)
        #pragma unroll
        for (int j = 0; j < NJ; ++j) acc[k][j][0] = acc[k][j][1] = 0.0;
    const double* row = Slots::at(sm.rows, gid, a.U + e * B5);
    if (!rows_landed<true>(bar, parity, a.err)) return false;
    const double gm1 = a.gamma - 1.0;
    #pragma unroll 1
    for (int nt = 0; nt < NT; ++nt) {
        double H[2][3][5];  // per point: the flux to integrate, direction by direction, in physical directions
        {
            double V[5][2], G[3][5][2];
            gradients8<NB>(V, G, row, a.t.tv + nt * KT * 32, A.v.tvd + nt * KT * 96, lane);
            #pragma unroll
            for (int i = 0; i < 2; ++i) {
                double X[5][3], Uv[5];
                #pragma unroll
                for (int k = 0; k < 5; ++k) {
                    Uv[k] = V[k][i];
                    #pragma unroll
                    for (int m = 0; m < 3; ++m) X[k][m] = J[3 * m] * G[0][k][i] + J[3 * m + 1] * G[1][k][i] + J[3 * m + 2] * G[2][k][i];
                }
                const ViscState st = visc_state(Uv);
                visc_flux_3(st, A.mu, A.cq, X, H[i]);
                if (CONV) {  // G - H
                    const double rho = Phys<double>::positive(Uv[0]), ir = 1.0 / rho;
                    const double u[3] = {Uv[1] * ir, Uv[2] * ir, Uv[3] * ir};
                    const double p = gm1 * (Uv[4] - 0.5 * rho * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]));
                    #pragma unroll
                    for (int m = 0; m < 3; ++m) {
                        const double ru = rho * u[m];
                        H[i][m][0] = ru;
                        #pragma unroll
                        for (int c = 0; c < 3; ++c) H[i][m][1 + c] = ru * u[c] + (c == m ? p : 0.0) - H[i][m][1 + c];
                        H[i][m][4] = u[m] * (Uv[4] + p) - H[i][m][4];
                    }
                }
            }
        }
        // acc += -(J^T H detJ) (w dphi)
        #pragma unroll
        for (int d = 0; d < 3; ++d) {
            double g[5][2];
            #pragma unroll
            for (int i = 0; i < 2; ++i) {
                const bool pad = NQV % 8 != 0 && nt * 8 + 2 * tq + i >= NQV;
                #pragma unroll
                for (int k = K0; k < 5; ++k)
                    g[k][i] = pad ? 0.0 : -detj * (J[d] * H[i][0][k] + J[3 + d] * H[i][1][k] + J[6 + d] * H[i][2][k]);
            }
            const double* tb = a.t.tw + (nt * 3 + d) * 2 * NJ * 32 + lane;
            #pragma unroll
            for (int i = 0; i < 2; ++i)
                #pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    const double b = __ldg(tb + (i * NJ + j) * 32);
                    #pragma unroll
                    for (int k = K0; k < 5; ++k) dmma884(acc[k][j], g[k][i], b);
                }
        }
    }
    #pragma unroll 1
    for (int q = 0; q < 4; ++q) {
        const int meta = grp.meta[q];
        const double sgn = (meta >> 8) ? -1.0 : 1.0;
        const double* rec = a.rec + (int64_t)grp.face[gid][q] * RW;
        const double* tb = a.t.tl + (int64_t)(meta & 0xff) * KF * NJ * 32 + lane;
        double m[5][KF];
        #pragma unroll
        for (int t = 0; t < KF; t += 2) {
            const int m0 = moment_of(NB, t, tq);
            #pragma unroll
            for (int k = K0; k < 5; ++k) {
                if (t + 1 < KF) {
                    double2 x = make_double2(0.0, 0.0);
                    if (8 * (t / 2) + 8 <= MR || m0 < MR) x = __ldcg(reinterpret_cast<const double2*>(rec + k * MR + m0));
                    m[k][t] = sgn * x.x;
                    m[k][t + 1] = sgn * x.y;
                } else {
                    m[k][t] = m0 < MR ? sgn * __ldcg(rec + k * MR + m0) : 0.0;
                }
            }
        }
        #pragma unroll
        for (int t = 0; t < KF; ++t)
            #pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const double b = __ldg(tb + (t * NJ + j) * 32);
                #pragma unroll
                for (int k = K0; k < 5; ++k) dmma884(acc[k][j], m[k][t], b);
            }
        #pragma unroll
        for (int j = 0; j < NJ; ++j)
            if (8 * j + 2 * tq < NB) {
                const double2 x = __ldcg(reinterpret_cast<const double2*>(rec + 5 * MR + 8 * j + 2 * tq));
                acc[4][j][0] = fma(sgn, x.x, acc[4][j][0]);
                acc[4][j][1] = fma(sgn, x.y, acc[4][j][1]);
            }
    }
    __syncwarp();
    const double* row0 = Slots::at(sm.rows0, gid, a.U0 + e * B5);
    double* os = Slots::at(sm.rows, gid, a.out + e * B5);
    const double sdt = CONV ? (a.dt_inst ? __ldg(a.dt_inst + __ldg(a.elem_inst + e)) : a.dt) * __ldg(a.inv_detj + e) : 0.0;
    #pragma unroll
    for (int j = 0; j < NJ; ++j)
        #pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int b = 8 * j + 2 * tq + i;  // mode
            if (b >= NB) continue;
            const double s = CONV ? sdt * __ldg(a.t.inv_mass + b) : 0.0;
            #pragma unroll
            for (int k = 0; k < 5; ++k) {
                if (CONV) {
                    const double x = row[5 * b + k] - s * acc[k][j][i];
                    os[5 * b + k] = u0 ? fma(a.a1, x, a.a0 * row0[5 * b + k]) : a.a1 * x;
                } else {
                    os[5 * b + k] = acc[k][j][i];
                }
            }
        }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    Slots::store(sm.rows, lane, n, a.out + (int64_t)grp.e[lane & 7] * B5);
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    __syncwarp();
    return true;
}

template <int NB, int NQV, bool CONV, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 1) visc_element_rows8(Visc8Args A) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint64_t bars[WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto& sm = reinterpret_cast<ElemSmem8<NB>*>(smem_raw)[warp];
    if (lane == 0) mbar_init(&bars[warp], 16);
    __syncwarp();
    unsigned parity = 0;
    for (int gi = blockIdx.x + gridDim.x * warp + await_previous(); gi < A.e.ngroups; gi += gridDim.x * WARPS) {
        if (gi + gridDim.x * WARPS >= A.e.ngroups) release_next();
        if (!visc_element_group8<NB, NQV, CONV>(A, gi, sm, bars[warp], parity, lane)) break;
    }
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

}  // namespace fvedg
