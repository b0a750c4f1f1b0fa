// FP64 kernels for rows of eight items (faces or elements): one warp per group, one tile of the FP64 tensor
// cores (mma m8n8k4) per conserved variable, row = item.
//
// As in the mixed form's groups of sixteen, a lane's accumulators of the five tiles hold all five variables of
// one item at the same two points (row gid, columns 2 tq and 2 tq + 1), so the fluxes are evaluated on the
// accumulators, and a result register is the next product's A operand as it stands: the contraction over the
// points runs its k-tiles over {2 tq} and {2 tq + 1}, in which order the tables are stored. Every row of a tile
// is an item, and a table fragment serves five products.
//
// Face fluxes are stored as moments on the triangle's polynomial basis (face_moments in dg_kernels_mixed16.cuh):
// formed once per face, contracted by both its elements.
//
// The FP64 pipe does a DMMA (256 FMAs) in 16 cycles and a DFMA (32) in 2, so both kernels are bound by the FP64
// operations themselves; what is not one of them has to fit beside.
#pragma once
#include <cstdint>

#include "dg_flux.cuh"
#include "dg_kernels_fp64.cuh"
#include "dg_kernels_mixed16.cuh"
#include "dg_launch.cuh"
#include "dg_slots.cuh"

namespace fvedg {

constexpr int kRows8 = 8;

struct alignas(16) FaceGroup8 {  // faces with equal (perm0, perm1, kind); unused slots repeat f[0]
    int f[kRows8];
    int n;
    int pad[3];
};
struct alignas(16) ElemGroup8 {  // elements with equal face maps in canonical face order; unused slots repeat slot 0
    int e[kRows8];
    int face[kRows8][4];
    int meta[4];
    int n;
    int pad[3];
};

// Moments of a variable in a face's record, padded to whole 16-byte units; their k-tiles: pairs of tiles over
// eight moments (columns 2 tq, then 2 tq + 1), and for a remainder of at most four one tile (column tq).
__host__ __device__ constexpr int moment_row(int nb) { return (face_moments(nb) + 1) / 2 * 2; }
__host__ __device__ constexpr int moment_ktiles(int nb) {
    return moment_row(nb) / 8 * 2 + (moment_row(nb) % 8 == 0 ? 0 : moment_row(nb) % 8 <= 4 ? 1 : 2);
}
// The moment that column tq of k-tile t holds (moment_row(nb) or more: none).
__host__ __device__ constexpr int moment_of(int nb, int t, int tq) {
    return t / 2 * 8 + (t == moment_ktiles(nb) - 1 && t % 2 == 0 ? tq : 2 * tq + t % 2);
}

struct Rows8Tables {
    const double* tf;        // [24][point tile][k-tile][lane]  phi_f: mode 4 kt + tq at point 8 nt + gid
    const double* tm;        // [point tile][i][moment tile][lane]  w psi: point 8 nt + 2 tq + i, moment 8 mt + gid
    const double* tv;        // [point tile][k-tile][lane]  phi_v
    const double* tw;        // [point tile][direction][i][mode tile][lane]  w dphi: point 8 nt + 2 tq + i, mode 8 j + gid
    const double* tl;        // [24][k-tile][mode tile][lane]  T[perm]: moment moment_of(kt, tq), mode 8 j + gid
    const double* mv;        // [mode tile][lane]  -sum_g w dphi: mode 8 j + gid, direction tq
    const double* inv_mass;  // [NB]
};

struct Rows8FaceArgs {
    const double* U;
    const FaceInfo* fi;
    const FaceGroup8* groups;
    int ngroups;
    const double* UD;        // Dirichlet data [nface][nqf][5] or null
    double* rec;             // [nface][5][moment_row]
    Rows8Tables t;
    double gamma;
    int flux;
    int faces_mask;          // bit 0: interior faces, bit 1: boundary faces
    int* err;
};

struct Rows8ElemArgs {
    const double* U;         // stage input
    const double* U0;        // U^n
    double* out;             // R (mode 0) or the new stage (mode 1)
    const double* rec;
    const double* jd;        // [ncell][9] det J * J^-T, row-major (c, d)
    const double* inv_detj;  // [ncell]
    const ElemGroup8* groups;
    int ngroups;
    Rows8Tables t;
    double gamma;
    int with_volume;
    int mode;
    double dt, a0, a1;       // out = a0 U0 + a1 (U - dt R / b)
    const double* dt_inst;
    const int* elem_inst;
    int* err;
};

// Slot strides for the A operand's reads (eight rows, columns 40 bytes apart): 32 or 96 (mod 128) touches every
// bank once.
constexpr int slot_stride8(int bytes) { return bytes % 128 == 32 || bytes % 128 == 96 ? bytes : slot_stride8(bytes + 16); }
template <int NB>
using Slots8 = RowSlotsOf<NB, slot_stride8((40 * NB + 8 + 15) / 16 * 16)>;

// P5 sums 94 x 3 products per mode in one accumulator and a face's 36 x 21 after them, and each product rounds at the
// size of what is there already: residuals were 5 to 12 % further from the exact ones than those of the scalar kernels.
// There the volume term is taken of the deviations from the mean state's flux (its own integral is one product), and
// the sums of a point tile's moments and of a face are formed by themselves: 8 to 17 % closer than the scalar kernels,
// 0.203 -> 0.220 ms a residual at 7,986 cells (scalar 0.585).
__host__ __device__ constexpr bool short_sums8(int nb) { return nb > 35; }

// The five variables at the points 8 nt + 2 tq + {0, 1} of the lane's row: v[k] += sum_b c_b phi_b, with the row
// in shared memory and the table's point tile at tb.
template <int NB>
__device__ __forceinline__ void values8(double (&v)[5][2], const double* row, const double* __restrict__ tb, int lane) {
    constexpr int KT = (NB + 3) / 4;
    const int tq = lane & 3;
    #pragma unroll
    for (int kt = 0; kt < KT; ++kt) {
        const double b = __ldg(tb + kt * 32 + lane);
        const bool on = 4 * kt + 3 < NB || 4 * kt + tq < NB;
        #pragma unroll
        for (int k = 0; k < 5; ++k) dmma884(v[k], on ? row[5 * (4 * kt + tq) + k] : 0.0, b);
    }
}

// ---- faces -----------------------------------------------------------------------------------------
template <int NB>
struct alignas(16) FaceSmem8 {
    unsigned char rows[2 * kRows8 * Slots8<NB>::BYTES];  // cells[0] of the eight faces, then cells[1]
};

template <int NB, int NQF>
__device__ __forceinline__ bool face_group8(const Rows8FaceArgs& a, int gi, FaceSmem8<NB>& sm, uint64_t& bar,
                                            unsigned& parity, int lane) {
    using Slots = Slots8<NB>;
    constexpr int B5 = 5 * NB, NT = pad8(NQF) / 8, KT = (NB + 3) / 4, MR = moment_row(NB), MT = (MR + 7) / 8;
    const int gid = lane >> 2, tq = lane & 3;
    const FaceGroup8& grp = a.groups[gi];
    const int n = grp.n, f = grp.f[gid];
    const FaceInfo F = a.fi[f];
    const int bc = (F.meta >> 16) & 0xff;
    const bool interior = F.c1 >= 0;
    const bool active = interior ? (a.faces_mask & 1)
                                 : ((a.faces_mask & 2) && ((bc == 0 && a.UD != nullptr) || bc == 5));
    if (!active) {
        for (int i = lane; i < n * 5 * MR; i += 32) a.rec[(int64_t)grp.f[i / (5 * MR)] * (5 * MR) + i % (5 * MR)] = 0.0;
        return true;
    }
    {   // lane i < 16 moves the row of cells[i / 8] of face i % 8 (a boundary face's one cell twice)
        const FaceInfo& mine = a.fi[grp.f[lane & 7]];
        const int c = (lane & 8) && interior ? mine.c1 : mine.c0;
        Slots::load(sm.rows, lane, 16, a.U + (int64_t)c * B5, &bar);
    }
    const double* left = Slots::at(sm.rows, gid, a.U + (int64_t)F.c0 * B5);
    const double* right = interior ? Slots::at(sm.rows, gid + 8, a.U + (int64_t)F.c1 * B5) : left;
    const double* tl = a.t.tf + (int64_t)(F.meta & 0xff) * NT * KT * 32;
    const double* tr = a.t.tf + (int64_t)((F.meta >> 8) & 0xff) * NT * KT * 32;
    double mom[5][MT][2];
    #pragma unroll
    for (int k = 0; k < 5; ++k)
        #pragma unroll
        for (int mt = 0; mt < MT; ++mt) mom[k][mt][0] = mom[k][mt][1] = 0.0;
    if (!rows_landed(bar, parity, a.err)) return false;
    #pragma unroll 1
    for (int nt = 0; nt < NT; ++nt) {
        double L[5][2], R[5][2];
        #pragma unroll
        for (int k = 0; k < 5; ++k) L[k][0] = L[k][1] = R[k][0] = R[k][1] = 0.0;
        values8<NB>(L, left, tl + nt * KT * 32, lane);
        if (interior) values8<NB>(R, right, tr + nt * KT * 32, lane);
        #pragma unroll
        for (int i = 0; i < 2; ++i) {
            double UL[5], UR[5], Fh[5];
            #pragma unroll
            for (int k = 0; k < 5; ++k) { UL[k] = L[k][i]; UR[k] = R[k][i]; }
            const int g = nt * 8 + 2 * tq + i;
            const bool pad = NQF % 8 != 0 && g >= NQF;
            if (!interior) {
                if (bc == 0) {  // Dirichlet ghost 2 U_D - U_in (ExplicitConvection.cpp:53)
                    const double* ud = a.UD + ((int64_t)f * NQF + (pad ? 0 : g)) * 5;
                    #pragma unroll
                    for (int k = 0; k < 5; ++k) UR[k] = ud[k] + (ud[k] - UL[k]);
                } else {        // Pseudo3DZ mirror (:92)
                    #pragma unroll
                    for (int k = 0; k < 5; ++k) UR[k] = UL[k];
                    UR[3] = -UL[3];
                }
            }
            if (a.flux == 1) roe_f64(UL, UR, F.n, a.gamma, Fh);
            else lax_friedrichs_f64(UL, UR, F.n, a.gamma, Fh);
            #pragma unroll
            for (int k = 0; k < 5; ++k) L[k][i] = pad ? 0.0 : Fh[k];
        }
        if constexpr (short_sums8(NB)) {
            #pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
                double part[5][2] = {};
                #pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const double b = __ldg(a.t.tm + ((nt * 2 + i) * MT + mt) * 32 + lane);
                    #pragma unroll
                    for (int k = 0; k < 5; ++k) dmma884(part[k], L[k][i], b);
                }
                #pragma unroll
                for (int k = 0; k < 5; ++k) { mom[k][mt][0] += part[k][0]; mom[k][mt][1] += part[k][1]; }
            }
        } else {
            #pragma unroll
            for (int i = 0; i < 2; ++i)
                #pragma unroll
                for (int mt = 0; mt < MT; ++mt) {
                    const double b = __ldg(a.t.tm + ((nt * 2 + i) * MT + mt) * 32 + lane);
                    #pragma unroll
                    for (int k = 0; k < 5; ++k) dmma884(mom[k][mt], L[k][i], b);
                }
        }
    }
    __syncwarp();  // the slots are free
    if (gid < n) {
        double* rec = a.rec + (int64_t)f * (5 * MR);
        #pragma unroll
        for (int mt = 0; mt < MT; ++mt)
            if (8 * mt + 2 * tq < MR)
                #pragma unroll
                for (int k = 0; k < 5; ++k)
                    *reinterpret_cast<double2*>(rec + k * MR + 8 * mt + 2 * tq) = make_double2(mom[k][mt][0] * F.jw, mom[k][mt][1] * F.jw);
    }
    return true;
}

// Bound by the FP64 pipe (65 % busy at P3: 42 % DMMA, 23 % the Roe solver's 163 operations a point) and by the
// latency of dependent products beside it. Per launch at P3, 384,000 tets: 0.682 ms in groups of three, 0.678 here;
// what it gains is the record, 400 bytes a face instead of 960. P1 0.308 -> 0.165 ms, P5 with the pair.
template <int NB, int NQF, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 1) face_flux_rows8(Rows8FaceArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint64_t bars[WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto& sm = reinterpret_cast<FaceSmem8<NB>*>(smem_raw)[warp];
    if (lane == 0) mbar_init(&bars[warp], 16);
    __syncwarp();
    unsigned parity = 0;
    for (int gi = blockIdx.x + gridDim.x * warp + await_previous(); gi < a.ngroups; gi += gridDim.x * WARPS) {
        if (gi + gridDim.x * WARPS >= a.ngroups) release_next();
        if (!face_group8<NB, NQF>(a, gi, sm, bars[warp], parity, lane)) break;
    }
}

// ---- elements --------------------------------------------------------------------------------------
template <int NB>
struct alignas(16) ElemSmem8 {
    unsigned char rows[kRows8 * Slots8<NB>::BYTES];   // the stage input, then the output
    unsigned char rows0[kRows8 * Slots8<NB>::BYTES];  // U^n
    ElemGroup8 grp;
    double mean[short_sums8(NB) ? kRows8 : 1][15];  // [item][direction, variable]: the mean state's flux
};

template <int NB, int NQV>
__device__ __forceinline__ bool element_group8(const Rows8ElemArgs& a, int gi, ElemSmem8<NB>& sm, uint64_t& bar,
                                               unsigned& parity, int lane) {
    using Slots = Slots8<NB>;
    constexpr int B5 = 5 * NB, NT = pad8(NQV) / 8, KT = (NB + 3) / 4, NJ = pad8(NB) / 8, MR = moment_row(NB);
    constexpr int KF = moment_ktiles(NB);
    constexpr bool SHORT = short_sums8(NB);
    const int gid = lane >> 2, tq = lane & 3;
    if (lane < (int)(sizeof(ElemGroup8) / 16))
        reinterpret_cast<uint4*>(&sm.grp)[lane] = __ldg(reinterpret_cast<const uint4*>(a.groups + gi) + lane);
    __syncwarp();
    const ElemGroup8& grp = sm.grp;
    const int n = grp.n;
    const int64_t e = grp.e[gid];
    const bool u0 = a.mode != 0 && a.a0 != 0.0;
    {   // lane i < 8: the stage input's row i; lane 8 + i: U^n's
        const int64_t mine = grp.e[lane & 7];
        Slots::load(sm.rows, lane, 8, a.U + mine * B5, &bar);
        if (lane >= 8 && lane < 16) {
            if (u0) Slots::load(sm.rows0, lane - 8, 8, a.U0 + mine * B5, &bar);
            else mbar_arrive(&bar);
        }
    }
    {   // the face records into L2 while the volume term is computed
        constexpr int NL = (5 * MR * 8 + 127) / 128;
        for (int i = lane; i < 4 * kRows8 * NL; i += 32) {
            const int fq = i / NL, part = i - fq * NL;
            prefetch_l2(reinterpret_cast<const char*>(a.rec + (int64_t)grp.face[fq >> 2][fq & 3] * (5 * MR)) + min(part * 128, 5 * MR * 8 - 8));
        }
    }
    double J[9];
    if (a.with_volume)
        #pragma unroll
        for (int i = 0; i < 9; ++i) J[i] = __ldg(a.jd + e * 9 + i);
    double acc[5][NJ][2];
    #pragma unroll
    for (int k = 0; k < 5; ++k)
        #pragma unroll
        for (int j = 0; j < NJ; ++j) acc[k][j][0] = acc[k][j][1] = 0.0;
    const double* row = Slots::at(sm.rows, gid, a.U + e * B5);
    if (!rows_landed(bar, parity, a.err)) return false;
    if (a.with_volume) {
        const double gm1 = a.gamma - 1.0;
        if constexpr (SHORT) {
            const double rho = Phys<double>::positive(row[0]), ir = 1.0 / rho;
            const double u[3] = {row[1] * ir, row[2] * ir, row[3] * ir};
            const double p = gm1 * (row[4] - 0.5 * rho * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]));
            if (tq < 3) {
                const double j0 = __ldg(a.jd + e * 9 + tq), j1 = __ldg(a.jd + e * 9 + 3 + tq), j2 = __ldg(a.jd + e * 9 + 6 + tq);
                const double v = u[0] * j0 + u[1] * j1 + u[2] * j2, rv = rho * v;
                double* g = sm.mean[gid] + 5 * tq;
                g[0] = rv;
                g[1] = rv * u[0] + p * j0;
                g[2] = rv * u[1] + p * j1;
                g[3] = rv * u[2] + p * j2;
                g[4] = (row[4] + p) * v;
            }
            __syncwarp();
        }
        #pragma unroll 1
        for (int nt = 0; nt < NT; ++nt) {
            double U[5][2], vel[3][2], p[2];
            #pragma unroll
            for (int k = 0; k < 5; ++k) U[k][0] = U[k][1] = 0.0;
            values8<NB>(U, row, a.t.tv + nt * KT * 32, lane);
            #pragma unroll
            for (int i = 0; i < 2; ++i) {
                U[0][i] = Phys<double>::positive(U[0][i]);
                const double ir = 1.0 / U[0][i];
                #pragma unroll
                for (int c = 0; c < 3; ++c) vel[c][i] = U[1 + c][i] * ir;
                p[i] = gm1 * (U[4][i] - 0.5 * U[0][i] * (vel[0][i] * vel[0][i] + vel[1][i] * vel[1][i] + vel[2][i] * vel[2][i]));
                U[4][i] += p[i];  // E + p
            }
            // -G = -(det J F J^-T), direction by direction: with v = u . J_d, G_0 = rho v, G_i = rho u_i v + p J_id,
            // G_4 = (E + p) v; acc += (-G) (w dphi): the volume term enters R with a minus
            // (ExplicitConvection.cpp:190-196)
            #pragma unroll
            for (int d = 0; d < 3; ++d) {
                double g[5][2];
                #pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const double v = vel[0][i] * J[d] + vel[1][i] * J[3 + d] + vel[2][i] * J[6 + d];
                    const double rv = U[0][i] * v;
                    if constexpr (SHORT) {
                        const double* b = sm.mean[gid] + 5 * d;
                        g[0][i] = b[0] - rv;
                        #pragma unroll
                        for (int c = 0; c < 3; ++c) g[1 + c][i] = fma(-p[i], J[3 * c + d], fma(-rv, vel[c][i], b[1 + c]));
                        g[4][i] = fma(-U[4][i], v, b[4]);
                    } else {
                        g[0][i] = -rv;
                        #pragma unroll
                        for (int c = 0; c < 3; ++c) g[1 + c][i] = -(rv * vel[c][i] + p[i] * J[3 * c + d]);
                        g[4][i] = -U[4][i] * v;
                    }
                    if (NQV % 8 != 0 && nt * 8 + 2 * tq + i >= NQV)  // a padding point
                        #pragma unroll
                        for (int k = 0; k < 5; ++k) g[k][i] = 0.0;
                }
                const double* tb = a.t.tw + (nt * 3 + d) * 2 * NJ * 32 + lane;
                #pragma unroll
                for (int i = 0; i < 2; ++i)
                    #pragma unroll
                    for (int j = 0; j < NJ; ++j) {
                        const double b = __ldg(tb + (i * NJ + j) * 32);
                        #pragma unroll
                        for (int k = 0; k < 5; ++k) dmma884(acc[k][j], g[k][i], b);
                    }
            }
        }
    }
    if (SHORT && a.with_volume) {  // the mean state's flux
        double m[5];
        #pragma unroll
        for (int k = 0; k < 5; ++k) m[k] = tq < 3 ? sm.mean[gid][5 * tq + k] : 0.0;
        #pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const double b = __ldg(a.t.mv + j * 32 + lane);
            #pragma unroll
            for (int k = 0; k < 5; ++k) dmma884(acc[k][j], m[k], b);
        }
    }
    // face integrals: + on cells[0], - on cells[1] (ExplicitConvection.cpp:247-266)
    #pragma unroll 1
    for (int q = 0; q < 4; ++q) {
        const int meta = grp.meta[q];
        const double sgn = (meta >> 8) ? -1.0 : 1.0, smom = SHORT ? 1.0 : sgn;  // on the moments, or on the face's sum
        const double* rec = a.rec + (int64_t)grp.face[gid][q] * (5 * MR);
        const double* tb = a.t.tl + (int64_t)(meta & 0xff) * KF * NJ * 32 + lane;
        double m[5][KF];
        #pragma unroll
        for (int t = 0; t < KF; t += 2) {
            const int m0 = moment_of(NB, t, tq);
            if (t + 1 < KF) {  // a pair of tiles: two consecutive moments
                #pragma unroll
                for (int k = 0; k < 5; ++k) {
                    double2 x = make_double2(0.0, 0.0);
                    if (8 * (t / 2) + 8 <= MR || m0 < MR) x = __ldcg(reinterpret_cast<const double2*>(rec + k * MR + m0));
                    m[k][t] = smom * x.x;
                    m[k][t + 1] = smom * x.y;
                }
            } else {
                #pragma unroll
                for (int k = 0; k < 5; ++k) m[k][t] = m0 < MR ? smom * __ldcg(rec + k * MR + m0) : 0.0;
            }
        }
        if constexpr (SHORT) {
            #pragma unroll
            for (int j = 0; j < NJ; ++j) {
                double part[5][2] = {};
                #pragma unroll
                for (int t = 0; t < KF; ++t) {
                    const double b = __ldg(tb + (t * NJ + j) * 32);
                    #pragma unroll
                    for (int k = 0; k < 5; ++k) dmma884(part[k], m[k][t], b);
                }
                #pragma unroll
                for (int k = 0; k < 5; ++k) {
                    acc[k][j][0] = fma(sgn, part[k][0], acc[k][j][0]);
                    acc[k][j][1] = fma(sgn, part[k][1], acc[k][j][1]);
                }
            }
        } else {
            #pragma unroll
            for (int t = 0; t < KF; ++t)
                #pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    const double b = __ldg(tb + (t * NJ + j) * 32);
                    #pragma unroll
                    for (int k = 0; k < 5; ++k) dmma884(acc[k][j], m[k][t], b);
                }
        }
    }
    // the update in the slots, ten consecutive DOFs per lane at a time; whole rows leave as bulk copies
    __syncwarp();
    const double* row0 = Slots::at(sm.rows0, gid, a.U0 + e * B5);
    double* os = Slots::at(sm.rows, gid, a.out + e * B5);
    const double sdt = a.mode ? (a.dt_inst ? __ldg(a.dt_inst + __ldg(a.elem_inst + e)) : a.dt) * __ldg(a.inv_detj + e) : 0.0;
    #pragma unroll
    for (int j = 0; j < NJ; ++j)
        #pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int b = 8 * j + 2 * tq + i;  // mode
            if (b >= NB) continue;
            if (a.mode == 0) {
                #pragma unroll
                for (int k = 0; k < 5; ++k) os[5 * b + k] = acc[k][j][i];
            } else {
                const double s = sdt * __ldg(a.t.inv_mass + b);
                #pragma unroll
                for (int k = 0; k < 5; ++k) {
                    const double x = row[5 * b + k] - s * acc[k][j][i];
                    os[5 * b + k] = u0 ? fma(a.a1, x, a.a0 * row0[5 * b + k]) : a.a1 * x;
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

// Bound by the FP64 pipe (72 % busy at P3, 64 % DMMA). Per launch at P3, 384,000 tets: 0.958 ms in groups of three,
// 0.547 here (16 of 16 rows instead of 15, ten moments a face instead of 24 points, 144 -> 52 k-tiles of loads);
// P2 Auto rules 0.644 -> 0.315 ms, P4 2.078 -> 1.531 ms.
template <int NB, int NQV, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 1) element_rows8(Rows8ElemArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint64_t bars[WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto& sm = reinterpret_cast<ElemSmem8<NB>*>(smem_raw)[warp];
    if (lane == 0) mbar_init(&bars[warp], 16);
    __syncwarp();
    unsigned parity = 0;
    for (int gi = blockIdx.x + gridDim.x * warp + await_previous(); gi < a.ngroups; gi += gridDim.x * WARPS) {
        if (gi + gridDim.x * WARPS >= a.ngroups) release_next();
        if (!element_group8<NB, NQV>(a, gi, sm, bars[warp], parity, lane)) break;
    }
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

}  // namespace fvedg
