// Mixed-precision kernels for groups of sixteen items (faces or elements): one warp per group, one
// MMA tile of 16 rows per conserved variable (row = item).
//
// With the variable as the tile and the item as the row, a lane's accumulators of the five tiles hold
// all five variables of the same items and quadrature points (rows gid and gid + 8, columns 2 tq and
// 2 tq + 1), so the pointwise flux is evaluated on the accumulators themselves, and its results already
// sit where the next contraction's A fragments want them (the D layout of an n-tile is the A layout of
// a k-tile). Nothing is transposed through shared memory, every row of the tile is an item, and one
// table fragment serves 80 rows instead of 15.
//
// The face fluxes reach the elements as moments: psi_m, m < NM, is a basis of the polynomials of
// degree P on the triangle, orthogonal under the face rule with psi_0 = 1. The trace of every mode lies
// in its span, phi_j(xi^perm) = sum_m T[perm][j][m] psi_m, so
//   sum_g w_g phi_j F(x_g) = sum_m T[perm][j][m] M_m,   M_m = sum_g w_g psi_m(x_g) F(x_g):
// the moments are formed once per face (NM = 10 instead of 24 point values at P3) and both its elements
// contract them. M_0 (the mode-0 face integral) is kept in FP64; the moments m >= 1 of the constant reference
// flux vanish, so they are moments of the deviation alone. The linear moments carry most of that deviation:
// they stay FP32 and enter with M_0 through the FP64 tensor cores, which keeps the error of the face
// integrals below that of contracting the point values themselves.
#pragma once
#include <cstring>

#include "dg_kernels_mixed.cuh"
#include "dg_slots.cuh"

namespace fvedg {

constexpr int kRows = 16;  // items per group

// Moments per face: the dimension of the degree-P polynomials on a triangle.
__host__ __device__ constexpr int face_moments(int nb) {
    return nb == 1 ? 1 : nb == 4 ? 3 : nb == 10 ? 6 : nb == 20 ? 10 : nb == 35 ? 15 : 21;
}
// A-row width of the moments m >= 3; the face kernel's tiles of moment columns (column x is m = x + 3, the
// linear moments m = 1, 2 come in the last two columns of the last tile but at P3, where they open a second).
__host__ __device__ constexpr int moment_cols(int nb) { return pad8(face_moments(nb) - 3); }
__host__ __device__ constexpr int moment_tiles(int nb) { return pad8(face_moments(nb) - 1) / 8; }
__host__ __device__ constexpr int linear_col(int nb) { return nb == 20 ? 8 : 8 * moment_tiles(nb) - 2; }

// Moment record of a face: words [0, 5 KM) five A rows of the moments m >= 3 (column m - 3), split BF16
// hi/lo in fragment order; then {M_1, M_2} of the five variables (FP32) and M_0 of the five (FP64).
// Whole 16-byte units.
__host__ __device__ constexpr int moment_rec_words(int nb) { return 5 * moment_cols(nb) + 20; }

struct alignas(16) FaceGroup16 {  // faces with equal (perm0, perm1, kind); unused slots repeat f[0]
    int f[kRows];
    int n;
    int pad[3];
};
struct alignas(16) ElemGroup16 {  // elements with equal face maps in canonical face order; unused slots repeat slot 0
    int e[kRows];
    int face[kRows][4];
    int meta[4];
    int n;
    int pad[3];
};

struct Mixed16Tables {
    const uint32_t* tfa;     // [24] B fragments of the traces: n = face point, k = mode (mode 0: zero)
    const uint32_t* tva;     // B fragments of the volume values: n = volume point, k = mode (mode 0: zero)
    const uint32_t* tvp;     // [point tile] B fragments of the volume integral: n = mode, k = 8 dir + point
    const uint32_t* tfm;     // [point tile][moment tile][lane] TF32 {hi, hi', lo, lo'} of w psi_m at points 2 tq, 2 tq + 1
    const uint32_t* tfl;     // [24] B fragments of the face integral: n = mode, k = m - 3, T[perm][j][m]
    const double* t0;        // [24][3][NB] T[perm][j][m], m < 3
    const double* mv;        // [NB][3] sum_g w_g dphi_j
    const float* wf;         // face weights, zero-padded to whole point tiles
    const double* inv_mass;  // [NB]
    double wsum;             // sum of the face weights
};

struct Mixed16FaceArgs {
    const double* U;
    const FaceInfo* fi;
    const FaceGroup16* groups;
    const double* UD;
    uint32_t* rec;           // [nface][moment_rec_words]
    Mixed16Tables t;
    int ngroups;
    float gamma;
    int flux;
    int faces_mask;
    int vec;                 // all state rows start on 16-byte boundaries
    int* err;                // status word in mapped host memory (DG_E_WATCHDOG when a bounded wait ran out), or null
};

struct Mixed16ElemArgs {
    const double* U;
    const double* U0;
    double* out;
    const uint32_t* rec;
    const double* geo;       // [ncell][10] J^-T row-major, detJ
    const ElemGroup16* groups;
    Mixed16Tables t;
    int ngroups;
    double gamma;
    int volume;              // 0: leave the volume term out
    double dt, a0, a1;
    int mode;                // 0: out = R; 1: out = a0 U0 + a1 (U - dt M^-1 R)
    const double* dt_inst;
    const int* elem_inst;
    const double* Rv;
    int vec;                 // all rows of U, U0 and out start on 16-byte boundaries
    int* err;
};

__device__ __forceinline__ uint4 ld_table4(const uint32_t* p) { return __ldg(reinterpret_cast<const uint4*>(p)); }
__device__ __forceinline__ uint2 ld_table2(const uint32_t* p) { return __ldg(reinterpret_cast<const uint2*>(p)); }

// Slots whose stride spreads the 16-byte accesses of the fragment pattern (eight rows, runs of 80 bytes) over
// all banks.
constexpr int slot_unit16(int u) { return u % 8 == 4 ? u : slot_unit16(u + 1); }
template <int NB>
using RowSlots = RowSlotsOf<NB, 16 * slot_unit16((40 * NB + 8 + 15) / 16)>;

// Ten consecutive doubles (two modes of five variables) of a slot; `two`: the second mode exists.
__device__ __forceinline__ void slot_pair(double (&d)[10], const double* p, bool vec, bool two) {
    if (vec) {
        #pragma unroll
        for (int i = 0; i < 5; ++i) {
            const double2 v = *reinterpret_cast<const double2*>(p + 2 * i);
            d[2 * i] = v.x;
            d[2 * i + 1] = v.y;
        }
    } else {
        #pragma unroll
        for (int i = 0; i < 10; ++i) d[i] = (i < 5 || two) ? p[i] : 0.0;
    }
}

// A operands of five variables from two rows in shared memory: tile k holds variable k, column x is mode x
// (the tables' mode-0 column is zero: only deviations are contracted). c0[row][k]: the mode-0 values.
template <int NB>
__device__ __forceinline__ void split_rows(AFrag<pad8(NB)> (&A)[5], float (&c0)[2][5], const double* r0,
                                           const double* r1, bool vec, int lane) {
    constexpr int K = pad8(NB), N16 = KTiles<K>::N16;
    const int tq = lane & 3;
    #pragma unroll
    for (int h = 0; h < K / 8; ++h) {  // column block [8 h, 8 h + 8)
        const int c = 8 * h + 2 * tq;
        #pragma unroll
        for (int r = 0; r < 2; ++r) {
            double d[10];
            if (8 * h + 8 <= NB || c < NB) {
                slot_pair(d, (r ? r1 : r0) + 5 * c, vec, c + 1 < NB);
            } else {
                #pragma unroll
                for (int i = 0; i < 10; ++i) d[i] = 0.0;
            }
            #pragma unroll
            for (int k = 0; k < 5; ++k) {
                const float x = (float)d[k], y = (float)d[5 + k];
                if (h == 0) c0[r][k] = __shfl_sync(0xffffffffu, x, lane & 28);
                if (h / 2 < N16) split2(x, y, A[k].h[h / 2][2 * (h & 1) + r], A[k].l[h / 2][2 * (h & 1) + r]);
                else split2(x, y, A[k].th[r], A[k].tl[r]);
            }
        }
    }
}

// x = hi + lo, both TF32 (11 significant bits; the low 13 bits of a word are zero).
__host__ __device__ __forceinline__ uint32_t tf32_cut(float x) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(x) & 0xffffe000u;
#else
    uint32_t u;
    std::memcpy(&u, &x, 4);
    return u & 0xffffe000u;
#endif
}
__device__ __forceinline__ void split_tf32(float x, uint32_t& hi, uint32_t& lo) {
    hi = tf32_cut(x);
    lo = tf32_cut(x - __uint_as_float(hi));
}
__device__ __forceinline__ void mma1688_tf32(float d[4], const uint32_t a[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// The five variables' values at the eight points of n-tile nt (deviations, without c0).
template <int K, bool Global = true>
__device__ __forceinline__ void values16(float (&v)[5][4], const AFrag<K> (&A)[5], const uint32_t* tb, int nt, int lane) {
    #pragma unroll
    for (int k = 0; k < 5; ++k)
        #pragma unroll
        for (int i = 0; i < 4; ++i) v[k][i] = 0.f;
    const uint32_t* tbn = tb + nt * KTiles<K>::NT_U32;
    #pragma unroll
    for (int t = 0; t < KTiles<K>::N16; ++t) {
        const uint32_t* at = tbn + t * 128 + lane * 4;
        const uint4 b = Global ? ld_table4(at) : *reinterpret_cast<const uint4*>(at);
        #pragma unroll
        for (int k = 0; k < 5; ++k) mma16816(v[k], A[k].h[t], b.x, b.y);
        #pragma unroll
        for (int k = 0; k < 5; ++k) mma16816(v[k], A[k].h[t], b.z, b.w);
        #pragma unroll
        for (int k = 0; k < 5; ++k) mma16816(v[k], A[k].l[t], b.x, b.y);
    }
    if constexpr (KTiles<K>::TAIL) {
        const uint32_t* at = tbn + KTiles<K>::N16 * 128 + lane * 2;
        const uint2 b = Global ? ld_table2(at) : *reinterpret_cast<const uint2*>(at);
        #pragma unroll
        for (int k = 0; k < 5; ++k) mma1688(v[k], A[k].th, b.x);
        #pragma unroll
        for (int k = 0; k < 5; ++k) mma1688(v[k], A[k].th, b.y);
        #pragma unroll
        for (int k = 0; k < 5; ++k) mma1688(v[k], A[k].tl, b.x);
    }
}

template <int NP>
struct alignas(16) Values16 {  // point values of a group: [variable][point tile][lane]
    float4 v[5][pad8(NP) / 8][32];
};

// ---- faces -----------------------------------------------------------------------------------------
template <int NB, int NQF>
struct alignas(16) FaceSmem16 {
    union {
        alignas(16) unsigned char rows[kRows * RowSlots<NB>::BYTES];  // one side's state rows
        Values16<NQF> trace[2];                                       // then both sides' traces
    };
};

// One group. The rows of its first side are in flight when it begins; those of its second side travel
// while the first side's traces are computed, and the next group's first side while its fluxes are.
// Returns false when a copy did not land within the poll limit (the status word is set).
template <int NB, int NQF>
__device__ __forceinline__ bool face_group16(const Mixed16FaceArgs& a, int gi, int next, FaceSmem16<NB, NQF>& sm,
                                             uint64_t& bar, unsigned& parity, int lane) {
    using Slots = RowSlots<NB>;
    constexpr int KB = pad8(NB), MF = pad8(NQF), NT = MF / 8, KM = moment_cols(NB), MT = moment_tiles(NB), LC = linear_col(NB);
    constexpr int RW = moment_rec_words(NB);
    const int gid = lane >> 2, tq = lane & 3;
    const FaceGroup16& grp = a.groups[gi];
    const int n = grp.n;
    const int f[2] = {grp.f[gid], grp.f[gid + 8]};
    const int meta = a.fi[f[0]].meta, bc = (meta >> 16) & 0xff;
    const bool interior = a.fi[f[0]].c1 >= 0;
    const bool active = interior ? (a.faces_mask & 1)
                                 : ((a.faces_mask & 2) && ((bc == 0 && a.UD != nullptr) || bc == 5));
    if (!active) {
        for (int i = lane; i < n * RW; i += 32) {
            const int r = i / RW;
            a.rec[(int64_t)grp.f[r] * RW + (i - r * RW)] = 0u;
        }
        // the rows in flight for it are let in, and the next group's sent for
        if (!rows_landed<true>(bar, parity, a.err)) return false;
        if (next >= 0) Slots::load(sm.rows, lane, kRows, a.U + (int64_t)a.fi[a.groups[next].f[lane & 15]].c0 * (5 * NB), &bar);
        return true;
    }
    auto landed = [&] { return rows_landed<true>(bar, parity, a.err); };
    // lane i < 16 moves row i: its cells in this group and the next
    const FaceInfo& mine = a.fi[grp.f[lane & 15]];
    const int right = mine.c1, more = next >= 0 ? a.groups[next].f[lane & 15] : -1;
    const int fc[2][2] = {{a.fi[f[0]].c0, a.fi[f[0]].c1}, {a.fi[f[1]].c0, a.fi[f[1]].c1}};
    float nv[2][3], jw[2], ref[2][5];
    AFrag<KB> A[5];
    float c0[2][5];
    auto side = [&](int s) {
        const double* r0 = a.U + (int64_t)fc[0][s] * (5 * NB);
        const double* r1 = a.U + (int64_t)fc[1][s] * (5 * NB);
        split_rows<NB>(A, c0, Slots::at(sm.rows, lane >> 2, r0), Slots::at(sm.rows, (lane >> 2) + 8, r1), a.vec, lane);
        __syncwarp();  // the slots are free
    };
    if (!landed()) return false;
    side(0);
    if (interior) Slots::load(sm.rows, lane, kRows, a.U + (int64_t)right * (5 * NB), &bar);
    #pragma unroll
    for (int r = 0; r < 2; ++r) {  // the reference flux: 2A F . n at c_0 of cells[0] (below: of both cells' mean flux)
        const FaceInfo& F = a.fi[f[r]];
        #pragma unroll
        for (int i = 0; i < 3; ++i) nv[r][i] = (float)F.n[i];
        jw[r] = (float)F.jw;
        float rho, vel[3], p;
        Phys<float>::flux_n(c0[r], nv[r], a.gamma - 1.f, ref[r], rho, vel, p);
    }
    float left[NT][5][4];
    #pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        values16<KB>(left[nt], A, a.t.tfa + (meta & 0xff) * NT * KTiles<KB>::NT_U32, nt, lane);
        #pragma unroll
        for (int k = 0; k < 5; ++k) {
            left[nt][k][0] += c0[0][k]; left[nt][k][1] += c0[0][k];
            left[nt][k][2] += c0[1][k]; left[nt][k][3] += c0[1][k];
        }
    }
    if (interior) {
        if (!landed()) return false;
        side(1);
    }
    #pragma unroll
    for (int nt = 0; nt < NT; ++nt)
        #pragma unroll
        for (int k = 0; k < 5; ++k)
            sm.trace[0].v[k][nt][lane] = make_float4(left[nt][k][0], left[nt][k][1], left[nt][k][2], left[nt][k][3]);
    if (interior) {
        const uint32_t* tb = a.t.tfa + ((meta >> 8) & 0xff) * NT * KTiles<KB>::NT_U32;
        #pragma unroll 1
        for (int nt = 0; nt < NT; ++nt) {
            float v[5][4];
            values16<KB>(v, A, tb, nt, lane);
            #pragma unroll
            for (int k = 0; k < 5; ++k)
                sm.trace[1].v[k][nt][lane] = make_float4(v[k][0] + c0[0][k], v[k][1] + c0[0][k], v[k][2] + c0[1][k], v[k][3] + c0[1][k]);
        }
    }
    #pragma unroll
    for (int r = 0; r < 2; ++r) {
        if (interior) {
            float g[5], rho, vel[3], p;
            Phys<float>::flux_n(c0[r], nv[r], a.gamma - 1.f, g, rho, vel, p);
            #pragma unroll
            for (int k = 0; k < 5; ++k) ref[r][k] = 0.5f * (ref[r][k] + g[k]);
        }
        #pragma unroll
        for (int k = 0; k < 5; ++k) ref[r][k] *= jw[r];
    }
    const int cnext = more >= 0 ? a.fi[more].c0 : 0;
    float mom[5][MT][4], m0[2][5];
    #pragma unroll
    for (int k = 0; k < 5; ++k) {
        m0[0][k] = m0[1][k] = 0.f;
        #pragma unroll
        for (int mt = 0; mt < MT; ++mt)
            #pragma unroll
            for (int i = 0; i < 4; ++i) mom[k][mt][i] = 0.f;
    }
    #pragma unroll 1
    for (int nt = 0; nt < NT; ++nt) {
        float d[5][4];  // flux deviations 2A F - ref
        #pragma unroll
        for (int r = 0; r < 2; ++r) {  // the two points of row gid + 8 r
            float2 UL[5], UR[5], Fh[5];
            #pragma unroll
            for (int k = 0; k < 5; ++k) UL[k] = reinterpret_cast<const float2*>(&sm.trace[0].v[k][nt][lane])[r];
            if (interior) {
                #pragma unroll
                for (int k = 0; k < 5; ++k) UR[k] = reinterpret_cast<const float2*>(&sm.trace[1].v[k][nt][lane])[r];
            } else if (bc == 0) {  // padding points read the last point's data; their weights are zero
                const int64_t g0 = min(nt * 8 + 2 * tq, NQF - 1), g1 = min(nt * 8 + 2 * tq + 1, NQF - 1);
                const double* u0 = a.UD + ((int64_t)f[r] * NQF + g0) * 5;
                const double* u1 = a.UD + ((int64_t)f[r] * NQF + g1) * 5;
                #pragma unroll
                for (int k = 0; k < 5; ++k)
                    UR[k] = make_float2((float)u0[k] + ((float)u0[k] - UL[k].x), (float)u1[k] + ((float)u1[k] - UL[k].y));
            } else {
                #pragma unroll
                for (int k = 0; k < 5; ++k) UR[k] = UL[k];
                UR[3] = make_float2(-UL[3].x, -UL[3].y);
            }
            if (a.flux == 1) roe_f32x2(UL, UR, nv[r], a.gamma, Fh);
            else lax_friedrichs_f32x2(UL, UR, nv[r], a.gamma, Fh);
            #pragma unroll
            for (int k = 0; k < 5; ++k) {
                const float2 x = fma2(Fh[k], f2(jw[r]), f2(-ref[r][k]));
                d[k][2 * r] = x.x;
                d[k][2 * r + 1] = x.y;
            }
        }
        const float2 w = __ldg(reinterpret_cast<const float2*>(a.t.wf + nt * 8 + 2 * tq));
        #pragma unroll
        for (int k = 0; k < 5; ++k)
            #pragma unroll
            for (int r = 0; r < 2; ++r) m0[r][k] = fmaf(w.x, d[k][2 * r], fmaf(w.y, d[k][2 * r + 1], m0[r][k]));
        {   // three TF32 products (22 bits; an 8-wide TF32 MMA costs what an 8-wide BF16 one does): column tq of
            // the tile is point 2 tq, column tq + 4 point 2 tq + 1, which is how the deviations sit
            uint4 b[MT];
            #pragma unroll
            for (int mt = 0; mt < MT; ++mt) b[mt] = ld_table4(a.t.tfm + (nt * MT + mt) * 128 + lane * 4);
            uint32_t hi[5][4], lo[5][4];
            #pragma unroll
            for (int k = 0; k < 5; ++k)
                #pragma unroll
                for (int i = 0; i < 4; ++i) split_tf32(d[k][(i & 1) * 2 + (i >> 1)], hi[k][i], lo[k][i]);
            #pragma unroll
            for (int mt = 0; mt < MT; ++mt) {
                #pragma unroll
                for (int k = 0; k < 5; ++k) mma1688_tf32(mom[k][mt], hi[k], b[mt].x, b[mt].y);
                #pragma unroll
                for (int k = 0; k < 5; ++k) mma1688_tf32(mom[k][mt], hi[k], b[mt].z, b[mt].w);
                #pragma unroll
                for (int k = 0; k < 5; ++k) mma1688_tf32(mom[k][mt], lo[k], b[mt].x, b[mt].y);
            }
        }
    }
    __syncwarp();  // the traces are done with
    if (more >= 0) Slots::load(sm.rows, lane, kRows, a.U + (int64_t)cnext * (5 * NB), &bar);
    // the record of rows gid and gid + 8
    #pragma unroll
    for (int r = 0; r < 2; ++r) {
        const bool on = gid + 8 * r < n;
        uint32_t* rec = a.rec + (int64_t)f[r] * RW;
        #pragma unroll
        for (int k = 0; k < 5; ++k) {
            uint32_t hi[2], lo[2];
            #pragma unroll
            for (int mt = 0; mt < KM / 8; ++mt) split2(mom[k][mt][2 * r], mom[k][mt][2 * r + 1], hi[mt], lo[mt]);
            if constexpr (KM == 16) {
                if (on) *reinterpret_cast<uint4*>(rec + k * KM + 4 * tq) = make_uint4(hi[0], hi[1], lo[0], lo[1]);
            } else if constexpr (KM == 8) {
                if (on) *reinterpret_cast<uint2*>(rec + k * KM + 2 * tq) = make_uint2(hi[0], lo[0]);
            }
        }
        float* lin = reinterpret_cast<float*>(rec + 5 * KM);
        if (on && tq == LC % 8 / 2) {
            constexpr int c = LC / 8;
            *reinterpret_cast<float4*>(lin) = make_float4(mom[0][c][2 * r], mom[0][c][2 * r + 1], mom[1][c][2 * r], mom[1][c][2 * r + 1]);
            *reinterpret_cast<float4*>(lin + 4) = make_float4(mom[2][c][2 * r], mom[2][c][2 * r + 1], mom[3][c][2 * r], mom[3][c][2 * r + 1]);
            *reinterpret_cast<float2*>(lin + 8) = make_float2(mom[4][c][2 * r], mom[4][c][2 * r + 1]);
        }
        // M_0 = ref sum_g w_g + sum_g w_g d_g, one number for both sides of the face (the quad's four lanes
        // hold it after the exchange; three of them store)
        double mean[5];
        #pragma unroll
        for (int k = 0; k < 5; ++k) {
            float s = m0[r][k];
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            mean[k] = (double)ref[r][k] * a.t.wsum + (double)s;
        }
        double* to = reinterpret_cast<double*>(rec + 5 * KM + 10);
        if (on && tq == 0) to[0] = mean[0];
        if (on && (tq == 1 || tq == 2))
            *reinterpret_cast<double2*>(to + 2 * tq - 1) = tq == 1 ? make_double2(mean[1], mean[2]) : make_double2(mean[3], mean[4]);
    }
    return true;
}

// Sends for the first side of a warp's first group.
template <int NB, int NQF>
__device__ __forceinline__ void face_begin16(const Mixed16FaceArgs& a, int gi, FaceSmem16<NB, NQF>& sm, uint64_t& bar, int lane) {
    RowSlots<NB>::load(sm.rows, lane, kRows, a.U + (int64_t)a.fi[a.groups[gi].f[lane & 15]].c0 * (5 * NB), &bar);
}

// Groups [g0, g1) of a warp, `step` apart.
template <int NB, int NQF>
__device__ __forceinline__ bool face_run16(const Mixed16FaceArgs& a, int g0, int g1, int step, FaceSmem16<NB, NQF>& sm,
                                           uint64_t& bar, unsigned& parity, int lane) {
    if (g0 < g1) face_begin16<NB, NQF>(a, g0, sm, bar, lane);
    for (int gi = g0; gi < g1; gi += step)
        if (!face_group16<NB, NQF>(a, gi, gi + step < g1 ? gi + step : -1, sm, bar, parity, lane)) return false;
    return true;
}

// Bound by instruction issue and dependence latency at three warps per scheduler (43 % of issue slots, 12 % of
// DRAM, 23 % of the tensor pipe at P3): 16 faces take 4,100 warp instructions, where groups of three took 9,200
// for as many. Measured per launch, Taylor-Green P3, 663,552 tets, Roe: 0.915 ms in groups of three, 0.767 ms
// here; density wave P2, 196,608 tets: 0.150, 0.098 ms; P4, 93,750 tets: 0.166, 0.167 ms. The slots and both
// sides' traces share 15 KB a warp, which is what lets twelve warps stay; with the second side's traces in
// registers at eight warps it took 1.04 ms, with the Riemann solver one point at a time 0.83 ms.
template <int NB, int NQF, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 1) face_flux_mixed16(Mixed16FaceArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint64_t bars[WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) mbar_init(&bars[warp], kRows);
    __syncwarp();
    unsigned parity = 0;
    face_run16<NB, NQF>(a, blockIdx.x * WARPS + warp + await_previous(), a.ngroups, gridDim.x * WARPS,
                        reinterpret_cast<FaceSmem16<NB, NQF>*>(smem_raw)[warp], bars[warp], parity, lane);
    if (NB <= 20) release_next();  // at P4 the next kernel's blocks took L1 from the last items (440 -> 467 us a step)
}

// ---- elements --------------------------------------------------------------------------------------
template <int NB, int NQV>
struct alignas(16) ElemSmem16 {
    using Slots = RowSlots<NB>;
    static constexpr int MR = 20;  // words of a record's M_0, M_1, M_2
    static constexpr size_t HALF = 8 * Slots::BYTES;
    union {  // the stage input's rows, then the point values; at the update eight rows of it and of U^n at a time
        alignas(16) unsigned char rows[2 * HALF];
        Values16<NQV> val;
    };
    union {
        uint32_t mean[4 * kRows][MR];  // M_0, M_1, M_2 of the group's faces, [4 row + q]; before that
        struct {
            float sGbf[kRows][15];
            float sJ[kRows][9];        // detJ J^-T
        };
    };
    double sGb[kRows][15];         // detJ F(c_0) J^-T (FP64)
    double sDT[kRows];             // dt / detJ
    double geo[kRows][10];         // J^-T, detJ
    ElemGroup16 grp[2];            // this group and the next
};

// All threads of the CTA copy `words` 32-bit words (a multiple of 4) into shared memory.
__device__ __forceinline__ uint32_t* stage_table(uint32_t* to, const uint32_t* from, int words) {
    for (int i = threadIdx.x; i < words / 4; i += blockDim.x)
        reinterpret_cast<uint4*>(to)[i] = __ldg(reinterpret_cast<const uint4*>(from) + i);
    return to + words;
}
// Words of an array of doubles, padded to whole 16-byte units.
__host__ __device__ constexpr int double_words(int n) { return (2 * n + 3) / 4 * 4; }
__device__ __forceinline__ uint32_t* stage_doubles(uint32_t* to, const double* from, int n) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) reinterpret_cast<double*>(to)[i] = __ldg(from + i);
    return to + double_words(n);
}

// Tables of the element kernel, in shared memory as far as they fit beside eight warps.
struct ElemTables16 {
    const uint32_t *tva, *tvp, *tfl;
    const double *t0, *mv, *inv_mass;
};
template <int NB, int NQV>
struct ElemSizes16 {
    static constexpr int NV = pad8(NQV) / 8, NJ = pad8(NB) / 8;
    static constexpr int TVA = NV * KTiles<pad8(NB)>::NT_U32, TVP = NV * NJ * KTiles<24>::NT_U32;
    static constexpr int TFL = 24 * NJ * (moment_cols(NB) / 8 * 64);
    static constexpr int DBL = double_words(72 * NB) + double_words(3 * NB) + double_words(NB);
    static constexpr size_t warp = sizeof(ElemSmem16<NB, NQV>);
    static constexpr bool shared = NB <= 20;
    static constexpr size_t tables = shared ? 4 * (size_t)(TVA + TVP + TFL + DBL) : 0;
};

// Sends for a group's record, and (once that is there) for its geometry; its state rows go to L2.
__device__ __forceinline__ void elem_record16(const Mixed16ElemArgs& a, int gi, ElemGroup16& grp, int lane) {
    if (lane < (int)(sizeof(ElemGroup16) / 16))
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(reinterpret_cast<uint4*>(&grp) + lane)),
                     "l"(reinterpret_cast<const uint4*>(a.groups + gi) + lane));
    asm volatile("cp.async.commit_group;");
}
template <int NB>
__device__ __forceinline__ void elem_geo16(const Mixed16ElemArgs& a, const ElemGroup16& grp, double (&geo)[kRows][10], int lane) {
    #pragma unroll
    for (int i = lane; i < kRows * 5; i += 32)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(&geo[i / 5][2 * (i % 5)])),
                     "l"(a.geo + (int64_t)grp.e[i / 5] * 10 + 2 * (i % 5)));
    asm volatile("cp.async.commit_group;");
    const double* row = (lane < kRows ? a.U : a.U0) + (int64_t)grp.e[lane & 15] * (5 * NB);
    if (lane < kRows || a.a0 != 0.0)
        #pragma unroll
        for (int o = 0; o < 40 * NB; o += 128) prefetch_l2(reinterpret_cast<const char*>(row) + min(o, 40 * NB - 8));
}

template <int NB, int NQV>
__device__ __forceinline__ bool element_group16(const Mixed16ElemArgs& a, const ElemTables16& t, int next, int turn,
                                                ElemSmem16<NB, NQV>& sm, uint64_t& bar, unsigned& parity,
                                                int lane) {
    using S = ElemSmem16<NB, NQV>;
    using Slots = RowSlots<NB>;
    constexpr int KB = pad8(NB), MV = pad8(NQV), MJ = pad8(NB), NJ = MJ / 8, KM = moment_cols(NB);
    constexpr int RW = moment_rec_words(NB), VW = KTiles<24>::NT_U32, B5 = 5 * NB, MR = S::MR;
    constexpr bool GL = !ElemSizes16<NB, NQV>::shared;
    auto tab4 = [](const uint32_t* p) { return GL ? ld_table4(p) : *reinterpret_cast<const uint4*>(p); };
    auto tab2 = [](const uint32_t* p) { return GL ? ld_table2(p) : *reinterpret_cast<const uint2*>(p); };
    const int gid = lane >> 2;
    const ElemGroup16& grp = sm.grp[turn];
    const int n = grp.n;
    const bool u0 = a.mode != 0 && a.a0 != 0.0;
    auto landed = [&] { return rows_landed<true>(bar, parity, a.err); };
    const int64_t mine = grp.e[lane & 15];  // lane i < 16 moves row i
    const bool more = next >= 0;
    if (more) elem_record16(a, next, sm.grp[turn ^ 1], lane);
    const double* ur[2] = {a.U + (int64_t)grp.e[gid] * B5, a.U + (int64_t)grp.e[gid + 8] * B5};
    Slots::load(sm.rows, lane, kRows, a.U + mine * B5, &bar);
    {   // the face records into L2
        constexpr int NL = (RW * 4 + 127) / 128;
        #pragma unroll
        for (int i = lane; i < 4 * kRows * NL; i += 32) {
            const int fq = i / NL, part = i - fq * NL;
            prefetch_l2(a.rec + (int64_t)grp.face[fq >> 2][fq & 3] * RW + min(32 * part, RW - 1));
        }
    }
    if (!landed()) return false;
    if (a.volume) {
        {
            AFrag<KB> A[5];
            float c0[2][5];
            split_rows<NB>(A, c0, Slots::at(sm.rows, gid, ur[0]), Slots::at(sm.rows, gid + 8, ur[1]), a.vec, lane);
            __syncwarp();
            #pragma unroll 1
            for (int nt = 0; nt < MV / 8; ++nt) {
                float v[5][4];
                values16<KB, !ElemSizes16<NB, NQV>::shared>(v, A, t.tva, nt, lane);
                #pragma unroll
                for (int k = 0; k < 5; ++k)
                    sm.val.v[k][nt][lane] = make_float4(v[k][0] + c0[0][k], v[k][1] + c0[0][k], v[k][2] + c0[1][k], v[k][3] + c0[1][k]);
            }
        }
        if (lane < kRows) {  // the flux of the mean state, one lane per element
            const double* geo = sm.geo[lane];
            const double* row = a.U + mine * B5;
            double c[5], J[9], Jf[9];
            #pragma unroll
            for (int i = 0; i < 5; ++i) c[i] = row[i];
            const double dj = geo[9];
            if (a.mode != 0)
                sm.sDT[lane] = (a.dt_inst ? __ldg(a.dt_inst + __ldg(a.elem_inst + mine)) : a.dt) * (1.0 / sm.geo[lane][9]);
            #pragma unroll
            for (int i = 0; i < 9; ++i) {
                J[i] = dj * geo[i];
                sm.sJ[lane][i] = (float)J[i];
                Jf[i] = (double)(float)J[i];
            }
            const double rho = c[0] > 1e-16 ? c[0] : 1e-16, ir = 1.0 / rho;
            const double u[3] = {c[1] * ir, c[2] * ir, c[3] * ir};
            const double p = (a.gamma - 1.0) * (c[4] - 0.5 * rho * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]));
            auto flux_d = [&](const double (&X)[9], int d, double (&g)[5]) {
                const double v = u[0] * X[d] + u[1] * X[3 + d] + u[2] * X[6 + d];
                g[0] = rho * v;
                #pragma unroll
                for (int i = 0; i < 3; ++i) g[1 + i] = rho * u[i] * v + p * X[3 * i + d];
                g[4] = (c[4] + p) * v;
            };
            // The points' fluxes are pulled back with the FP32 geometry, so the deviations are taken from the mean
            // state's flux pulled back with it too; what that differs from its FP32 value goes to the FP64 part. With
            // the exact flux rounded in its place every step had the same error of half an FP32 unit.
            #pragma unroll
            for (int d = 0; d < 3; ++d) {
                double g[5], gf[5];
                flux_d(J, d, g);
                flux_d(Jf, d, gf);
                #pragma unroll
                for (int k = 0; k < 5; ++k) {
                    const float r = (float)gf[k];
                    sm.sGb[lane][3 * k + d] = g[k] - (gf[k] - (double)r);
                    sm.sGbf[lane][3 * k + d] = r;
                }
            }
        }
        __syncwarp();
    }
    if (!a.volume) {
        if (lane < kRows) {
            #pragma unroll
            for (int i = 0; i < 15; ++i) sm.sGb[lane][i] = 0.0;
            if (a.mode != 0) {
                sm.sDT[lane] = (a.dt_inst ? __ldg(a.dt_inst + __ldg(a.elem_inst + mine)) : a.dt) * (1.0 / sm.geo[lane][9]);
            }
        }
        __syncwarp();
    }
    float acc[5][NJ][4];
    #pragma unroll
    for (int k = 0; k < 5; ++k)
        #pragma unroll
        for (int nt = 0; nt < NJ; ++nt)
            #pragma unroll
            for (int i = 0; i < 4; ++i) acc[k][nt][i] = 0.f;
    if (a.volume) {
        const float gm1 = (float)a.gamma - 1.f;
        #pragma unroll 1
        for (int nt = 0; nt < MV / 8; ++nt) {
            // row r of the lane's pair: both its points at once
            float2 U[5][2], np[2], mj[3][2], v[3][2];
            #pragma unroll
            for (int k = 0; k < 5; ++k) {
                const float4 x = sm.val.v[k][nt][lane];
                U[k][0] = make_float2(x.x, x.y);
                U[k][1] = make_float2(x.z, x.w);
            }
            // Gb - G per direction d: with v = u . J_d, G_0 = m . J_d, G_i = m_i v + p J_id, G_4 = (E + p) v;
            // one variable at a time, directions 0 and 1 as one 16-wide k-tile, direction 2 as an 8-wide one. The
            // momentum's pressure comes last: taken from Gb first, it left a rounding that is the same at all points
            // of a flow of one pressure, and 200 steps of a density wave (P2) were 20 % further off.
            #pragma unroll
            for (int r = 0; r < 2; ++r) {
                const float2 ir = rcp2(max2(U[0][r], 1e-16f));
                float2 vel[3];
                #pragma unroll
                for (int c = 0; c < 3; ++c) vel[c] = mul2(U[1 + c][r], ir);
                const float2 ke = fma2(vel[2], U[3][r], fma2(vel[1], U[2][r], mul2(vel[0], U[1][r])));
                const float2 p = mul2(f2(gm1), fma2(f2(-0.5f), ke, U[4][r]));
                U[4][r] = add2(U[4][r], p);  // E + p
                np[r] = mul2(p, f2(-1.f));
                const float* J = sm.sJ[gid + 8 * r];
                #pragma unroll
                for (int d = 0; d < 3; ++d) {  // -m . J_d, -v
                    mj[d][r] = fma2(U[1][r], f2(-J[d]), fma2(U[2][r], f2(-J[3 + d]), mul2(U[3][r], f2(-J[6 + d]))));
                    v[d][r] = mul2(mj[d][r], ir);
                }
            }
            const uint32_t* tb = t.tvp + nt * NJ * VW;
            uint4 b01[NJ];
            uint2 b2[NJ];
            #pragma unroll
            for (int j = 0; j < NJ; ++j) {
                b01[j] = tab4(tb + j * VW + lane * 4);
                b2[j] = tab2(tb + j * VW + 128 + lane * 2);
            }
            // two variables at a time: six accumulators apart, an MMA finds the one before it finished
            #pragma unroll
            for (int k0 = 0; k0 < 5; k0 += 2) {
                constexpr int KS = 2;
                uint32_t h[KS][6], l[KS][6];  // [direction][row]
                #pragma unroll
                for (int kk = 0; kk < KS; ++kk) {
                    const int k = k0 + kk;
                    if (k > 4) continue;
                    #pragma unroll
                    for (int d = 0; d < 3; ++d)
                        #pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            const float* J = sm.sJ[gid + 8 * r] + d;
                            const float2 gb = f2(sm.sGbf[gid + 8 * r][3 * k + d]);
                            float2 g;
                            if (k == 0) g = add2(gb, mj[d][r]);
                            else if (k < 4) g = fma2(np[r], f2(J[3 * (k - 1)]), fma2(U[k][r], v[d][r], gb));
                            else g = fma2(U[4][r], v[d][r], gb);
                            split2(g.x, g.y, h[kk][2 * d + r], l[kk][2 * d + r]);
                        }
                }
                auto each = [&](auto&& mma) {
                    #pragma unroll
                    for (int kk = 0; kk < KS; ++kk)
                        #pragma unroll
                        for (int j = 0; j < NJ; ++j)
                            if (k0 + kk < 5) mma(acc[k0 + kk][j], kk, j);
                };
                each([&](float(&c)[4], int kk, int j) { mma16816(c, h[kk], b01[j].x, b01[j].y); });
                each([&](float(&c)[4], int kk, int j) { mma16816(c, h[kk], b01[j].z, b01[j].w); });
                each([&](float(&c)[4], int kk, int j) { mma16816(c, l[kk], b01[j].x, b01[j].y); });
                each([&](float(&c)[4], int kk, int j) { mma1688(c, h[kk] + 4, b2[j].x); });
                each([&](float(&c)[4], int kk, int j) { mma1688(c, h[kk] + 4, b2[j].y); });
                each([&](float(&c)[4], int kk, int j) { mma1688(c, l[kk] + 4, b2[j].x); });
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();  // the volume term is done with its shared memory; the next group's record is there
    {   // M_0, M_1, M_2 of the 64 faces, past L1 (a record may be new in this launch)
        constexpr int MU = MR / 4;
        #pragma unroll
        for (int i = lane; i < 4 * kRows * MU; i += 32) {
            const int fq = i / MU, part = i - fq * MU;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(&sm.mean[fq][4 * part])),
                         "l"(a.rec + (int64_t)grp.face[fq >> 2][fq & 3] * RW + 5 * KM + 4 * part));
        }
        asm volatile("cp.async.commit_group;");
    }
    if (more) elem_geo16<NB>(a, sm.grp[turn ^ 1], sm.geo, lane);
    // the update works on eight rows at a time: their stage input and U^n
    auto fetch = [&](int r) {  // rows [8 r, 8 r + 8)
        const int64_t el = grp.e[(lane & 7) + 8 * r];
        Slots::load(sm.rows, lane, 8, a.U + el * B5, &bar);
        if (lane >= 8 && lane < 16) {
            if (u0) Slots::load(sm.rows + S::HALF, lane - 8, 8, a.U0 + el * B5, &bar);
            else mbar_arrive(&bar);
        }
    };
    if (a.mode != 0) fetch(0);
    // face integrals of the moments m >= 3; side 1 negated exactly. The tensor cores cut a sum to FP32 instead of
    // rounding it, in proportion to what is in the accumulator already: at P2, where the errors add up the most, each
    // face is summed by itself and added to the volume term by a rounding addition (density wave, 200 steps: 8 % less
    // error; the kernel is no slower. At P3 and P4 it cost 0.7 % and the errors are below those of groups of three).
    constexpr bool SUMS = NB == 10;
    if constexpr (KM > 0) {
        #pragma unroll 1
        for (int q = 0; q < 4; ++q) {
            AFrag<KM> F[5];
            const uint32_t flip = (grp.meta[q] >> 8) ? 0x80008000u : 0u;
            const uint32_t* r0 = a.rec + (int64_t)grp.face[gid][q] * RW;
            const uint32_t* r1 = a.rec + (int64_t)grp.face[gid + 8][q] * RW;
            #pragma unroll
            for (int k = 0; k < 5; ++k) load_afrag<KM>(F[k], r0 + k * KM, r1 + k * KM, lane, flip);
            const uint32_t* tb = t.tfl + (grp.meta[q] & 0xff) * NJ * KTiles<KM>::NT_U32;
            #pragma unroll
            for (int j = 0; j < NJ; ++j) {
                float part[5][4] = {};
                if constexpr (KM == 16) {
                    const uint4 b = tab4(tb + j * KTiles<KM>::NT_U32 + lane * 4);
                    #pragma unroll
                    for (int k = 0; k < 5; ++k) mma16816(SUMS ? part[k] : acc[k][j], F[k].h[0], b.x, b.y);
                    #pragma unroll
                    for (int k = 0; k < 5; ++k) mma16816(SUMS ? part[k] : acc[k][j], F[k].h[0], b.z, b.w);
                    #pragma unroll
                    for (int k = 0; k < 5; ++k) mma16816(SUMS ? part[k] : acc[k][j], F[k].l[0], b.x, b.y);
                } else {
                    const uint2 b = tab2(tb + j * KTiles<KM>::NT_U32 + lane * 2);
                    #pragma unroll
                    for (int k = 0; k < 5; ++k) mma1688(SUMS ? part[k] : acc[k][j], F[k].th, b.x);
                    #pragma unroll
                    for (int k = 0; k < 5; ++k) mma1688(SUMS ? part[k] : acc[k][j], F[k].th, b.y);
                    #pragma unroll
                    for (int k = 0; k < 5; ++k) mma1688(SUMS ? part[k] : acc[k][j], F[k].tl, b.x);
                }
                if (SUMS) {
                    #pragma unroll
                    for (int k = 0; k < 5; ++k)
                        #pragma unroll
                        for (int i = 0; i < 4; ++i) acc[k][j][i] += part[k][i];
                }
            }
        }
    }
    // FP64 parts on the FP64 tensor cores in the accumulators' layout: the four faces' M_0, M_1, M_2 with
    // +-T[perm][j][m] and the mean flux with -mv, K = 16. Then the update in the slots, ten consecutive DOFs per lane at
    // a time, and the finished rows leave as bulk copies.
    int ln = lane;
    asm volatile("" : "+r"(ln));  // keeps its index arithmetic inside the group loop
    const int row0 = ln >> 2, tq = ln & 3;
    const int mq = grp.meta[tq];
    const double sq = (mq >> 8) ? -1.0 : 1.0;
    const double* t0 = t.t0 + (mq & 0xff) * 3 * NB;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    #pragma unroll
    for (int r = 0; r < 2; ++r) {
        if (a.mode != 0 && !landed()) return false;
        const int row = row0 + 8 * r;
        const int64_t base = (int64_t)grp.e[row] * B5;
        const double* am = reinterpret_cast<const double*>(sm.mean[4 * row + tq] + 10);
        const float* lin = reinterpret_cast<const float*>(sm.mean[4 * row + tq]);
        const double* us = Slots::at(sm.rows, row0, a.U + base);
        const double* vs = Slots::at(sm.rows + S::HALF, row0, a.U0 + base);
        double* os = Slots::at(sm.rows, row0, a.out + base);
        const double sdt = a.mode != 0 ? sm.sDT[row] : 0.0;
        #pragma unroll
        for (int nt = 0; nt < NJ; ++nt) {
            const int jb = nt * 8 + row0;
            const double b0 = jb < NB ? sq * t0[jb] : 0.0, bu = jb < NB ? sq * t0[NB + jb] : 0.0, bv = jb < NB ? sq * t0[2 * NB + jb] : 0.0;
            const double b1 = (jb < NB && tq < 3) ? -t.mv[3 * jb + tq] : 0.0;
            const int j = nt * 8 + 2 * tq;  // this lane's modes j, j + 1
            const bool two = j + 1 < NB;
            double R[10];
            #pragma unroll
            for (int k = 0; k < 5; ++k) {
                double d[2];  // widened in place: hoisted together, the conversions would hold 120 registers
                asm volatile("cvt.f64.f32 %0, %1;" : "=d"(d[0]) : "f"(acc[k][nt][2 * r]));
                asm volatile("cvt.f64.f32 %0, %1;" : "=d"(d[1]) : "f"(acc[k][nt][2 * r + 1]));
                dmma884(d, am[k], b0);
                dmma884(d, (double)lin[2 * k], bu);
                dmma884(d, (double)lin[2 * k + 1], bv);
                dmma884(d, tq < 3 ? sm.sGb[row][3 * k + tq] : 0.0, b1);
                R[k] = d[0];
                R[5 + k] = d[1];
            }
            if (j < NB) {
                if (a.Rv) {
                    #pragma unroll
                    for (int i = 0; i < 10; ++i)
                        if (i < 5 || two) R[i] -= a.Rv[base + 5 * j + i];
                }
                if (a.mode != 0) {
                    double u[10], v[10];
                    slot_pair(u, us + 5 * j, a.vec, two);
                    if (u0) slot_pair(v, vs + 5 * j, a.vec, two);
                    const double s0 = __dmul_rn(sdt, t.inv_mass[j]), s1 = two ? __dmul_rn(sdt, t.inv_mass[j + 1]) : 0.0;
                    #pragma unroll
                    for (int i = 0; i < 10; ++i) R[i] = rk_update(u0, a.a0, u0 ? v[i] : 0.0, a.a1, u[i], i < 5 ? s0 : s1, R[i]);
                }
                if (a.vec) {
                    #pragma unroll
                    for (int i = 0; i < 5; ++i) *reinterpret_cast<double2*>(os + 5 * j + 2 * i) = make_double2(R[2 * i], R[2 * i + 1]);
                } else {
                    #pragma unroll
                    for (int i = 0; i < 10; ++i)
                        if (i < 5 || two) os[5 * j + i] = R[i];
                }
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        const int64_t el = grp.e[(ln & 7) + 8 * r];
        Slots::store(sm.rows, ln, min(8, n - 8 * r), a.out + el * B5);
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        __syncwarp();
        if (r == 0 && a.mode != 0) fetch(1);
    }
    return true;
}

// A warp's first group: record and geometry, in slot 0.
template <int NB, int NQV>
__device__ __forceinline__ void elem_begin16(const Mixed16ElemArgs& a, int gi, ElemSmem16<NB, NQV>& sm, int lane) {
    elem_record16(a, gi, sm.grp[0], lane);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    elem_geo16<NB>(a, sm.grp[0], sm.geo, lane);
}

// Groups [g0, g1) of a warp, `step` apart.
template <int NB, int NQV>
__device__ __forceinline__ bool elem_run16(const Mixed16ElemArgs& a, const ElemTables16& t, int g0, int g1, int step,
                                           ElemSmem16<NB, NQV>& sm, uint64_t& bar, unsigned& parity, int lane) {
    if (g0 < g1) elem_begin16<NB, NQV>(a, g0, sm, lane);
    bool ok = true;
    int turn = 0;
    for (int gi = g0; gi < g1 && ok; gi += step, turn ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
        ok = element_group16<NB, NQV>(a, t, gi + step < g1 ? gi + step : -1, turn, sm, bar, parity, lane);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    return ok;
}

// The element kernel's tables into shared memory (all threads of the CTA), or their global addresses.
template <int NB, int NQV>
__device__ __forceinline__ ElemTables16 elem_tables16(const Mixed16Tables& g, unsigned char* smem) {
    using S = ElemSizes16<NB, NQV>;
    ElemTables16 t{g.tva, g.tvp, g.tfl, g.t0, g.mv, g.inv_mass};
    if constexpr (S::shared) {
        uint32_t* tab = reinterpret_cast<uint32_t*>(smem);
        t.tva = tab;
        t.tvp = tab = stage_table(tab, g.tva, S::TVA);
        t.tfl = tab = stage_table(tab, g.tvp, S::TVP);
        tab = stage_table(tab, g.tfl, S::TFL);
        t.t0 = reinterpret_cast<const double*>(tab);
        tab = stage_doubles(tab, g.t0, 72 * NB);
        t.mv = reinterpret_cast<const double*>(tab);
        tab = stage_doubles(tab, g.mv, 3 * NB);
        t.inv_mass = reinterpret_cast<const double*>(tab);
        stage_doubles(tab, g.inv_mass, NB);
    }
    return t;
}

// Bound by dependence latency at two warps per scheduler (28 % of issue slots, 36 % of DRAM, 24 % of the tensor
// pipe at P3): 16 elements take 5,000 warp instructions, where groups of three took 14,000 for as many. Per
// launch, as above: P3 1.071 ms in groups of three, 0.700 ms here; P2 0.211, 0.146 ms; P4 0.352, 0.270 ms. Rows
// come and go as bulk copies: read by the lanes in fragment order they cost half a sector per access and the L1
// that the tables need (0.75 ms); staged through registers they spilled (1.05 ms). Tables next to the rows in
// shared memory up to P3: left to the 4 KB of L1 that remain, every n-tile waited for L2 (0.83 ms).
template <int NB, int NQV, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 1) element_mixed16(Mixed16ElemArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint64_t bars[WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const ElemTables16 t = elem_tables16<NB, NQV>(a.t, smem_raw);
    if (lane == 0) mbar_init(&bars[warp], kRows);
    __syncthreads();
    unsigned parity = 0;
    elem_run16<NB, NQV>(a, t, blockIdx.x * WARPS + warp + await_previous(), a.ngroups, gridDim.x * WARPS,
                        reinterpret_cast<ElemSmem16<NB, NQV>*>(smem_raw + ElemSizes16<NB, NQV>::tables)[warp],
                        bars[warp], parity, lane);
    if (NB <= 20) release_next();
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// Warps of a kernel's one CTA per SM: what shared memory holds (1 KB is the system's, and the barriers are
// static), at most `most`.
__host__ __device__ constexpr int warps16(int most, size_t warp_smem, size_t tables = 0) {
    const int fit = (int)((231936 - tables) / warp_smem);
    return fit < most ? fit : most;
}

}  // namespace fvedg
