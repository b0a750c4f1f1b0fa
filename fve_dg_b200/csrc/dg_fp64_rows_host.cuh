// Host side of the FP64 kernels for rows of eight: tables in fragment order, groups and buffers.
#pragma once
#include <vector>

#include "dg_fp64_rows.h"
#include "dg_mixed_host.cuh"
#include "dg_status.cuh"
#include "dg_viscous_rows.h"

namespace fvedg {

struct Rows8Data {
    bool ready = false;
    int order = 0, qv = 0, qf = 0;
    int nfgroups = 0, negroups = 0;
    int sms = 148;
    uint32_t maps = 0;  // the face maps (bit p) that the mesh has: a box of cubes has a third of the 24
    std::vector<void*> bufs;
    Rows8Tables t{};
    const FaceGroup8* fgroups = nullptr;
    const ElemGroup8* egroups = nullptr;
    const double* jd = nullptr;
    const double* inv_detj = nullptr;
    double* rec = nullptr;  // [nface][5][moment_row(nb)]
    int* err = nullptr;  // status word in mapped host memory, the context's
};

inline bool rows8_supported(int order, int qv, int qf) {
#define X(P, QV, QF, NB, NQV, NQF) \
    if (order == P && qv == QV && qf == QF) return true;
    FVEDG_ROWS8_COMBOS(X)
#undef X
    return false;
}

template <typename T>
inline int rows8_upload(Rows8Data& m, const T** dst, const std::vector<T>& v) {
    void* p = nullptr;
    if (cudaMalloc(&p, sizeof(T) * std::max<size_t>(v.size(), 1)) != cudaSuccess) return DG_E_NOMEM;
    m.bufs.push_back(p);
    if (!v.empty() && cudaMemcpy(p, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice) != cudaSuccess)
        return DG_E_CUDA;
    *dst = (const T*)p;
    return DG_OK;
}

// Whether the convective operator of a mesh of that many cells runs in rows of eight. Orders 0 and 5 have no other
// tensor-core kernels and take them at any size, if the groups are full enough (rows8_groups; P0 56 -> 39 us a step at n = 4 against the runtime-size kernels, P5
// 326 -> 233; n = 24: 372 -> 260 and 16,345 -> 4,838). For the others groups of three are the faster on small meshes,
// where a warp's chain of work decides (us a step, three / eight: P1 31 / 36 at n = 8, 34 / 36 at n = 9, 42 / 40 at
// n = 11; P2 54 / 54 at n = 6, 60 / 56 at n = 8, 64 / 58 at n = 9; P3 68 / 74, 80 / 79, 93 / 81; P4 103 / 127, 131 / 134,
// 177 / 140): five groups per SM at P1, about 6,000 cells, three above.
inline bool rows8_convective(int order, int qv, int64_t nowned, int sms) {
    const int per_sm = order == 0 || order == 5 ? 0 : order == 1 ? 5 : 3;
    if (nowned < (int64_t)per_sm * kRows8 * sms) return false;
    // P4 has eight warps per SM: with the 44-point rule a second round of groups that is less than a fifth full costs
    // more than it saves (10,368 cells: 283 us a step in threes, 298 in eights; 57 points: 354, 337)
    const int64_t round = (int64_t)kRows8 * 8 * sms;
    return !(order == 4 && qv == 5 && nowned > round && nowned * 5 < round * 6);
}

// The groups of eight, and whether they are full enough to use: a mesh with many classes of face maps (node orders of
// cells and faces as another program lists them) leaves as many partial groups, each as costly as a full one, and takes
// the other kernels at any size; orders 0 and 5 then take the scalar ones.
inline bool rows8_groups(int order, int qv, int qf, const std::vector<FaceInfo>& hfi, const std::vector<ElemFace>& hef,
                         int64_t nowned, std::vector<FaceGroup8>& fg, std::vector<ElemGroup8>& eg) {
    if (!rows8_supported(order, qv, qf)) return false;
    int inner = 0;
    build_groups(hfi, hef, nowned, fg, eg, &inner);
    return (int64_t)eg.size() * kRows8 * 3 <= nowned * 4 && (int64_t)fg.size() * kRows8 * 3 <= (int64_t)hfi.size() * 4;
}

// det J * J^-T and 1 / det J of the cells from their geometry ([10]: J^-T, det J).
__global__ void rows8_geometry(const double* __restrict__ geo, int64_t ncell, double* __restrict__ jd, double* __restrict__ inv_detj) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 10 * ncell) return;
    const int64_t e = i / 10;
    const int k = (int)(i - 10 * e);
    if (k < 9) jd[9 * e + k] = geo[10 * e + 9] * geo[i];
    else inv_detj[e] = 1.0 / geo[i];
}

inline uint32_t face_maps_of(const std::vector<FaceInfo>& hfi) {
    uint32_t maps = 0;
    for (const FaceInfo& f : hfi) maps |= 1u << (f.meta & 0xff) | (f.c1 >= 0 ? 1u << (f.meta >> 8 & 0xff) : 0u);
    return maps;
}

// The tables of the face maps in m.maps. geo: the cells' geometry on the device. m.jd and m.inv_detj, if set, are the same of another set of kernels.
inline int init_rows8(Rows8Data& m, const Tables& tab, const double* geo, const std::vector<FaceGroup8>& fg,
                      const std::vector<ElemGroup8>& eg, int64_t ncell, int64_t nface, int qv, int qf,
                      bool with_records = true) {
    const int NB = tab.nb, NQV = tab.nqv, NQF = tab.nqf, NM = face_moments(NB), MR = moment_row(NB);
    const int KT = (NB + 3) / 4, NF = pad8(NQF) / 8, NV = pad8(NQV) / 8, NJ = pad8(NB) / 8, MT = (MR + 7) / 8;
    const int KF = moment_ktiles(NB);
    m.order = tab.order; m.qv = qv; m.qf = qf;
    std::vector<double> psi, norm, T, tf, tm, tv, tw, tl;
    face_moment_basis(tab.order, qf, psi, norm);
    face_moment_maps(tab, qf, psi, norm, T, m.maps);
    tf.assign((size_t)24 * NF * KT * 32, 0.0);
    tw.reserve((size_t)NV * 6 * NJ * 32);
    tl.assign((size_t)24 * KF * NJ * 32, 0.0);
    for (int p = 0; p < 24; ++p)
        for (int nt = 0; nt < NF && (m.maps >> p & 1u); ++nt)
            for (int kt = 0; kt < KT; ++kt)
                for (int l = 0; l < 32; ++l) {
                    const int g = 8 * nt + l / 4, b = 4 * kt + l % 4;
                    if (g < NQF && b < NB) tf[((size_t)(p * NF + nt) * KT + kt) * 32 + l] = tab.phi_f[((size_t)p * NQF + g) * NB + b];
                }
    for (int nt = 0; nt < NF; ++nt)
        for (int i = 0; i < 2; ++i)
            for (int mt = 0; mt < MT; ++mt)
                for (int l = 0; l < 32; ++l) {
                    const int g = 8 * nt + 2 * (l % 4) + i, k = 8 * mt + l / 4;
                    tm.push_back(g < NQF && k < NM ? tab.w_f[g] * psi[(size_t)k * NQF + g] : 0.0);
                }
    for (int nt = 0; nt < NV; ++nt)
        for (int kt = 0; kt < KT; ++kt)
            for (int l = 0; l < 32; ++l) {
                const int g = 8 * nt + l / 4, b = 4 * kt + l % 4;
                tv.push_back(g < NQV && b < NB ? tab.phi_v[(size_t)g * NB + b] : 0.0);
            }
    for (int nt = 0; nt < NV; ++nt)
        for (int d = 0; d < 3; ++d)
            for (int i = 0; i < 2; ++i)
                for (int j = 0; j < NJ; ++j)
                    for (int l = 0; l < 32; ++l) {
                        const int g = 8 * nt + 2 * (l % 4) + i, b = 8 * j + l / 4;
                        tw.push_back(g < NQV && b < NB ? tab.dphi_vw[((size_t)g * NB + b) * 3 + d] : 0.0);
                    }
    std::vector<double> mv;
    for (int j = 0; j < NJ && short_sums8(NB); ++j)
        for (int l = 0; l < 32; ++l) {
            const int b = 8 * j + l / 4, d = l % 4;
            long double s = 0;
            if (b < NB && d < 3)
                for (int g = 0; g < NQV; ++g) s -= tab.dphi_vw[((size_t)g * NB + b) * 3 + d];
            mv.push_back((double)s);
        }
    for (int p = 0; p < 24; ++p)
        for (int t = 0; t < KF && (m.maps >> p & 1u); ++t)
            for (int j = 0; j < NJ; ++j)
                for (int l = 0; l < 32; ++l) {
                    const int k = moment_of(NB, t, l % 4), b = 8 * j + l / 4;
                    if (k < NM && b < NB) tl[((size_t)(p * KF + t) * NJ + j) * 32 + l] = T[((size_t)p * NB + b) * NM + k];
                }
    std::vector<double> inv_mass(NB);
    for (int j = 0; j < NB; ++j) inv_mass[j] = 1.0 / tab.mass_ref[j];
    m.nfgroups = (int)fg.size();
    m.negroups = (int)eg.size();
    int rc;
    if ((rc = rows8_upload(m, &m.t.tf, tf)) || (rc = rows8_upload(m, &m.t.tm, tm)) || (rc = rows8_upload(m, &m.t.tv, tv)) ||
        (rc = rows8_upload(m, &m.t.tw, tw)) || (rc = rows8_upload(m, &m.t.tl, tl)) ||
        (rc = rows8_upload(m, &m.t.mv, mv)) || (rc = rows8_upload(m, &m.t.inv_mass, inv_mass)) || (rc = rows8_upload(m, &m.fgroups, fg)) ||
        (rc = rows8_upload(m, &m.egroups, eg)))
        return rc;
    if (!m.jd) {
        void* p = nullptr;
        if (cudaMalloc(&p, sizeof(double) * 10 * ncell) != cudaSuccess) return DG_E_NOMEM;
        m.bufs.push_back(p);
        double* jd = (double*)p;
        rows8_geometry<<<(unsigned)((10 * ncell + 255) / 256), 256>>>(geo, ncell, jd, jd + 9 * ncell);
        if ((rc = cuda_status(cudaGetLastError())) || (rc = cuda_status(cudaStreamSynchronize(0)))) return rc;
        m.jd = jd;
        m.inv_detj = jd + 9 * ncell;
    }
    if (with_records) {
        void* p = nullptr;
        const size_t n = sizeof(double) * nface * 5 * MR;
        if (cudaMalloc(&p, n) != cudaSuccess) return DG_E_NOMEM;
        m.bufs.push_back(p);
        if (cudaMemset(p, 0, n) != cudaSuccess) return DG_E_CUDA;
        m.rec = (double*)p;
    }
    m.ready = true;
    return DG_OK;
}

inline void free_rows8(Rows8Data& m) {
    for (void* p : m.bufs) cudaFree(p);
    m.bufs.clear();
    m.ready = false;
}

// The viscous operator in rows of eight: tables of the derivatives and face records; the tables, groups and
// status word it shares with the convective kernels are a context's own or built here.
struct Visc8Data {
    bool ready = false;
    Rows8Data own;               // built when the context has no Rows8Data
    const Rows8Data* rows = nullptr;
    Visc8Tables v{};
    double* rec = nullptr;       // [nface][visc_rec(nb)]
    std::vector<void*> bufs;
};

inline int init_visc8(Visc8Data& m, const Tables& tab, int64_t nface, int qf) {
    const int NB = tab.nb, NQV = tab.nqv, NQF = tab.nqf, NM = face_moments(NB);
    const int KT = (NB + 3) / 4, NF = pad8(NQF) / 8, NV = pad8(NQV) / 8, NJ = pad8(NB) / 8, KD = deriv_ktiles(NB);
    std::vector<double> psi, norm, tfd, tvd, td;
    face_moment_basis(tab.order, qf, psi, norm);
    const uint32_t maps = m.rows->maps;
    tfd.assign((size_t)24 * NF * KT * 96, 0.0);
    tvd.reserve((size_t)NV * KT * 96);
    td.assign((size_t)72 * KD * NJ * 32, 0.0);
    for (int p = 0; p < 24; ++p)
        for (int nt = 0; nt < NF && (maps >> p & 1u); ++nt)
            for (int kt = 0; kt < KT; ++kt)
                for (int d = 0; d < 3; ++d)
                    for (int l = 0; l < 32; ++l) {
                        const int g = 8 * nt + l / 4, b = 4 * kt + l % 4;
                        if (g < NQF && b < NB)
                            tfd[((size_t)((p * NF + nt) * KT + kt) * 3 + d) * 32 + l] = tab.dphi_f[(((size_t)p * NQF + g) * NB + b) * 3 + d];
                    }
    for (int nt = 0; nt < NV; ++nt)
        for (int kt = 0; kt < KT; ++kt)
            for (int d = 0; d < 3; ++d)
                for (int l = 0; l < 32; ++l) {
                    const int g = 8 * nt + l / 4, b = 4 * kt + l % 4;
                    tvd.push_back(g < NQV && b < NB ? tab.dphi_v[((size_t)g * NB + b) * 3 + d] : 0.0);
                }
    // D[perm][d][j][m] = sum_g w_g dphi_j,d psi_m / |psi_m|^2; zero for moments past the derivative's degree
    const std::vector<long double> w = moment_projection(qf, psi, norm);
    std::vector<double> D((size_t)3 * NB * NM), dphi((size_t)3 * NB * NQF);
    for (int p = 0; p < 24; ++p) {
        if (!(maps >> p & 1u)) continue;
        for (int g = 0; g < NQF; ++g)
            for (int i = 0; i < 3 * NB; ++i) dphi[(size_t)i * NQF + g] = tab.dphi_f[((size_t)p * NQF + g) * NB * 3 + i];
        for (int b = 0; b < NB; ++b) {
            const int deg = mode_degree(b), most = std::min(NM, deg * (deg + 1) / 2);
            for (int d = 0; d < 3; ++d)
                for (int k = 0; k < most; ++k) {
                    const double* x = &dphi[(size_t)(3 * b + d) * NQF];
                    long double s = 0, s2 = 0;
                    int g = 0;
                    for (; g + 1 < NQF; g += 2) {
                        s += w[(size_t)k * NQF + g] * x[g];
                        s2 += w[(size_t)k * NQF + g + 1] * x[g + 1];
                    }
                    if (g < NQF) s += w[(size_t)k * NQF + g] * x[g];
                    D[((size_t)d * NB + b) * NM + k] = (double)(s + s2);
                }
        }
        for (int d = 0; d < 3; ++d)
            for (int t = 0; t < KD; ++t)
                for (int j = 0; j < NJ; ++j)
                    for (int l = 0; l < 32; ++l) {
                        const int k = 8 * (t / 2) + 2 * (l % 4) + t % 2, b = 8 * j + l / 4;
                        if (k < NM && b < NB) td[((size_t)((p * 3 + d) * KD + t) * NJ + j) * 32 + l] = D[((size_t)d * NB + b) * NM + k];
                    }
    }
    auto up = [&](const double** dst, const std::vector<double>& v) {
        void* p = nullptr;
        if (cudaMalloc(&p, sizeof(double) * v.size()) != cudaSuccess) return (int)DG_E_NOMEM;
        m.bufs.push_back(p);
        *dst = (const double*)p;
        return cudaMemcpy(p, v.data(), sizeof(double) * v.size(), cudaMemcpyHostToDevice) == cudaSuccess ? (int)DG_OK : (int)DG_E_CUDA;
    };
    int rc;
    if ((rc = up(&m.v.tfd, tfd)) || (rc = up(&m.v.tvd, tvd)) || (rc = up(&m.v.td, td))) return rc;
    void* p = nullptr;
    if (cudaMalloc(&p, sizeof(double) * nface * visc_rec(NB)) != cudaSuccess) return DG_E_NOMEM;
    m.bufs.push_back(p);
    m.rec = (double*)p;
    m.ready = true;
    return DG_OK;
}

inline void free_visc8(Visc8Data& m) {
    free_rows8(m.own);
    for (void* p : m.bufs) cudaFree(p);
    m.bufs.clear();
    m.ready = false;
}

}  // namespace fvedg
