// Host side of the mixed-precision form: tables in fragment order, item groups, buffers and launches.
#pragma once
#include <cmath>
#include <cstdlib>

#include "dg_groups.h"
#include "dg_kernels_mixed.cuh"
#include "dg_mixed16.h"
#include "dg_mixed_combos.h"

namespace fvedg {

struct MixedData {
    // Large meshes run the kernels for groups of sixteen (dg_kernels_mixed16.cuh), small ones those for
    // groups of three; the group counts below are of the groups in use.
    bool wide = false;
    Mixed16Tables t16{};
    const FaceGroup16* fgroups16 = nullptr;
    const ElemGroup16* egroups16 = nullptr;
    uint32_t* rec = nullptr;          // moment records [nface][moment_rec_words(nb)]

    bool ready = false;
    int order = 0, qv = 0, qf = 0, nb = 0, nqv = 0, nqf = 0;
    int64_t ncell = 0, nface = 0;
    int nfgroups = 0, negroups = 0;
    int nfgroups_inner = 0;  // face groups [0, nfgroups_inner) touch no ghost element
    float gamma = 1.4f;
    int flux = 0;
    int sms = 148;
    std::vector<void*> bufs;
    MixedTables t{};
    const FaceInfo* fi = nullptr;
    const FaceGroup* fgroups = nullptr;
    const ElemGroup* egroups = nullptr;
    const double* geo = nullptr;
    const double* inv_detj = nullptr;
    const double* UD = nullptr;
    uint32_t* dev = nullptr;          // face records [nface][face_rec_words(nqf)]
    const double* dt_inst = nullptr;  // ensembles: per-instance dt (device), else null
    const int* elem_inst = nullptr;
    const double* Rv = nullptr;       // Navier-Stokes stepping: the stage input's viscous residual
    int* err = nullptr;               // status word of the mixed kernels (bounded waits), in mapped host memory
    // element kernel: 0 = loads phase by phase (8-warp CTAs, four per SM), 2 = each group's rows
    // staged by TMA bulk copies (P1..P3, 16-byte aligned state buffers); chosen by dg_autotune
    int elem_kernel = 0;
    int elem_ctas = 1;                // resident CTAs per SM of the staged kernel: 1 or 2
    // host copies the tile schedule of the persistent form is built from
    std::vector<FaceGroup> hfg;
    std::vector<ElemGroup> heg;
    std::vector<FaceGroup16> hfg16;
    std::vector<ElemGroup16> heg16;
    std::vector<int> hface_cells;  // [nface][2]
};

inline bool mixed_supported(int order, int qv, int qf) {
#define X(P, QV, QF, NB, NQV, NQF, W) \
    if (order == P && qv == QV && qf == QF) return true;
    FVEDG_MIXED_COMBOS(X)
#undef X
    return false;
}

template <typename T>
inline int mixed_upload(MixedData& m, const T** dst, const std::vector<T>& v) {
    void* p = nullptr;
    if (cudaMalloc(&p, sizeof(T) * std::max<size_t>(v.size(), 1)) != cudaSuccess) return DG_E_NOMEM;
    m.bufs.push_back(p);
    if (!v.empty() && cudaMemcpy(p, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice) != cudaSuccess)
        return DG_E_CUDA;
    *dst = (const T*)p;
    return DG_OK;
}

template <typename T>
inline int mixed_alloc(MixedData& m, T** dst, size_t n) {
    void* p = nullptr;
    if (cudaMalloc(&p, sizeof(T) * std::max<size_t>(n, 1)) != cudaSuccess) return DG_E_NOMEM;
    m.bufs.push_back(p);
    if (cudaMemset(p, 0, sizeof(T) * std::max<size_t>(n, 1)) != cudaSuccess) return DG_E_CUDA;
    *dst = (T*)p;
    return DG_OK;
}

// B operand of one contraction in fragment order. T is N x K row-major (N, K multiples of 8). Per
// n-tile: for each full K tile, 32 lanes x {hi(c,c+1), hi(c+8,c+9), lo(c,c+1), lo(c+8,c+9)} of
// row n = 8 nt + lane / 4, c = 16 t + 2 (lane % 4); then the tail, 32 lanes x {hi(c,c+1), lo(c,c+1)}.
inline void append_frag_table(const std::vector<double>& T, int N, int K, std::vector<uint32_t>& out) {
    const int n16 = K / 16;
    const bool tail = (K % 16) != 0;
    auto half = [&](int n, int k, bool lo) -> uint32_t {
        const float f = (float)T[(size_t)n * K + k];
        const __nv_bfloat16 h = __float2bfloat16_rn(f);
        return (uint32_t)__bfloat16_as_ushort(lo ? __float2bfloat16_rn(f - __bfloat162float(h)) : h);
    };
    auto word = [&](int n, int c, bool lo) { return half(n, c, lo) | (half(n, c + 1, lo) << 16); };
    for (int nt = 0; nt < N / 8; ++nt) {
        for (int t = 0; t < n16; ++t)
            for (int lane = 0; lane < 32; ++lane) {
                const int n = nt * 8 + lane / 4, c = t * 16 + 2 * (lane % 4);
                out.push_back(word(n, c, false));
                out.push_back(word(n, c + 8, false));
                out.push_back(word(n, c, true));
                out.push_back(word(n, c + 8, true));
            }
        if (tail)
            for (int lane = 0; lane < 32; ++lane) {
                const int n = nt * 8 + lane / 4, c = n16 * 16 + 2 * (lane % 4);
                out.push_back(word(n, c, false));
                out.push_back(word(n, c, true));
            }
    }
}

// A basis of the polynomials of degree <= order on the triangle, orthogonal under the face rule, with
// psi_0 = 1: monomials u^i v^j by degree, Gram-Schmidt (twice) in the rule's inner product, whose
// exactness makes it a true one up to that degree. psi[m][g], norm[m] = sum_g w_g psi_m^2.
inline void face_moment_basis(int order, int qf, std::vector<double>& psi, std::vector<double>& norm) {
    const int nq = tri_rule_npts(qf), nm = (order + 1) * (order + 2) / 2;
    const double* r = tri_rule(qf);
    std::vector<long double> p((size_t)nm * nq), nn(nm);
    int m = 0;
    for (int d = 0; d <= order; ++d)
        for (int j = 0; j <= d; ++j, ++m) {
            for (int g = 0; g < nq; ++g)
                p[(size_t)m * nq + g] = std::pow((long double)r[3 * g], d - j) * std::pow((long double)r[3 * g + 1], j);
            for (int pass = 0; pass < 2; ++pass)
                for (int l = 0; l < m; ++l) {
                    long double s = 0;
                    for (int g = 0; g < nq; ++g) s += (long double)r[3 * g + 2] * p[(size_t)m * nq + g] * p[(size_t)l * nq + g];
                    for (int g = 0; g < nq; ++g) p[(size_t)m * nq + g] -= s / nn[l] * p[(size_t)l * nq + g];
                }
            long double s = 0;
            for (int g = 0; g < nq; ++g) s += (long double)r[3 * g + 2] * p[(size_t)m * nq + g] * p[(size_t)m * nq + g];
            if (m > 0) {  // unit length relative to psi_0
                long double w = nn[0], c = std::sqrt(w / s);
                for (int g = 0; g < nq; ++g) p[(size_t)m * nq + g] *= c;
                s = w;
            }
            nn[m] = s;
        }
    psi.assign(p.begin(), p.end());
    norm.assign(nn.begin(), nn.end());
}

// Total degree of mode j of the basis on the tetrahedron, which is listed by degree (as the moments are).
inline int mode_degree(int j) {
    int d = 0;
    while (j >= (d + 1) * (d + 2) * (d + 3) / 6) ++d;
    return d;
}

// The projection onto the moments, w_g psi_m(g) / |psi_m|^2, [m][g].
inline std::vector<long double> moment_projection(int qf, const std::vector<double>& psi, const std::vector<double>& norm) {
    const int nq = tri_rule_npts(qf);
    const double* r = tri_rule(qf);
    std::vector<long double> w(psi.size());
    for (size_t m = 0; m < norm.size(); ++m)
        for (int g = 0; g < nq; ++g) w[m * nq + g] = (long double)r[3 * g + 2] * psi[m * nq + g] / norm[m];
    return w;
}

// T[perm][j][m] with phi_j(xi^perm_g) = sum_m T psi_m(g) at every face point; zero for moments of a higher degree
// than the mode's, and for face maps that are not in `maps`.
inline void face_moment_maps(const Tables& tab, int qf, const std::vector<double>& psi, const std::vector<double>& norm,
                             std::vector<double>& T, uint32_t maps = 0xffffffu) {
    const int nb = tab.nb, nq = tab.nqf, nm = (int)norm.size();
    const std::vector<long double> w = moment_projection(qf, psi, norm);
    T.assign((size_t)24 * nb * nm, 0.0);
    for (int p = 0; p < 24; ++p) {
        if (!(maps >> p & 1u)) continue;
        T[(size_t)p * nb * nm] = 1.0;  // phi_0 = psi_0 = 1
        for (int j = 1; j < nb; ++j) {
            const int d = mode_degree(j), most = std::min(nm, (d + 1) * (d + 2) / 2);
            const double* phi = &tab.phi_fT[((size_t)p * nb + j) * nq];
            for (int m = 0; m < most; ++m) {
                const long double* wm = &w[(size_t)m * nq];
                long double s = 0, s2 = 0;  // two chains, for the speed
                int g = 0;
                for (; g + 1 < nq; g += 2) {
                    s += wm[g] * phi[g];
                    s2 += wm[g + 1] * phi[g + 1];
                }
                if (g < nq) s += wm[g] * phi[g];
                T[((size_t)p * nb + j) * nm + m] = (double)(s + s2);
            }
        }
    }
}

// Tables, groups and records of the kernels for groups of sixteen.
inline int init_mixed16(MixedData& m, const Tables& tab, int64_t nface, int qf) {
    const int NB = tab.nb, NQV = tab.nqv, NQF = tab.nqf, NM = face_moments(NB);
    const int KB = pad8(NB), MF = pad8(NQF), MV = pad8(NQV), MJ = pad8(NB), KM = moment_cols(NB);
    std::vector<double> psi, norm, T;
    face_moment_basis(tab.order, qf, psi, norm);
    face_moment_maps(tab, qf, psi, norm, T);
    std::vector<uint32_t> ftfa, ftva, ftvp, ftfm, ftfl;
    std::vector<double> t0((size_t)72 * NB), mv((size_t)NB * 3, 0.0);
    for (int p = 0; p < 24; ++p) {
        std::vector<double> tfa((size_t)MF * KB, 0.0), tfl((size_t)MJ * KM, 0.0);
        for (int g = 0; g < NQF; ++g)
            for (int b = 1; b < NB; ++b) tfa[(size_t)g * KB + b] = tab.phi_f[((size_t)p * NQF + g) * NB + b];
        for (int j = 0; j < NB; ++j) {
            for (int k = 0; k < 3; ++k) t0[((size_t)p * 3 + k) * NB + j] = T[((size_t)p * NB + j) * NM + k];
            for (int k = 3; k < NM; ++k) tfl[(size_t)j * KM + k - 3] = T[((size_t)p * NB + j) * NM + k];
        }
        append_frag_table(tfa, MF, KB, ftfa);
        if (KM > 0) append_frag_table(tfl, MJ, KM, ftfl);
    }
    std::vector<double> tva((size_t)MV * KB, 0.0);
    for (int g = 0; g < NQV; ++g)
        for (int b = 1; b < NB; ++b) tva[(size_t)g * KB + b] = tab.phi_v[(size_t)g * NB + b];
    append_frag_table(tva, MV, KB, ftva);
    for (int t = 0; t < MV / 8; ++t) {  // per point tile: column 8 d + i is direction d of point 8 t + i
        std::vector<double> tvp((size_t)MJ * 24, 0.0);
        for (int j = 0; j < NB; ++j)
            for (int i = 0; i < 8 && 8 * t + i < NQV; ++i)
                for (int d = 0; d < 3; ++d) tvp[(size_t)j * 24 + 8 * d + i] = tab.dphi_vw[((size_t)(8 * t + i) * NB + j) * 3 + d];
        append_frag_table(tvp, MJ, 24, ftvp);
    }
    for (int j = 0; j < NB; ++j)
        for (int g = 0; g < NQV; ++g)
            for (int d = 0; d < 3; ++d) mv[j * 3 + d] += tab.dphi_vw[((size_t)g * NB + j) * 3 + d];
    for (int t = 0; t < MF / 8; ++t)
        for (int mt = 0; mt < moment_tiles(NB); ++mt)
            for (int lane = 0; lane < 32; ++lane) {
                const int x = 8 * mt + lane / 4, l = x - linear_col(NB);  // column: m = x + 3, or a linear moment
                const int m = l == 0 || l == 1 ? 1 + l : x < NM - 3 ? x + 3 : NM;
                uint32_t hi[2], lo[2];
                for (int i = 0; i < 2; ++i) {
                    const int g = 8 * t + 2 * (lane % 4) + i;
                    const double v = (m < NM && g < NQF) ? tab.w_f[g] * psi[(size_t)m * NQF + g] : 0.0;
                    hi[i] = tf32_cut((float)v);
                    float hf;
                    std::memcpy(&hf, &hi[i], 4);
                    lo[i] = tf32_cut((float)(v - hf));
                }
                for (uint32_t w : {hi[0], hi[1], lo[0], lo[1]}) ftfm.push_back(w);
            }
    std::vector<float> wf(MF, 0.f);
    for (int g = 0; g < NQF; ++g) wf[g] = (float)tab.w_f[g];
    m.t16.wsum = m.t.wsum;
    m.t16.inv_mass = m.t.inv_mass;
    int rc;
    if ((rc = mixed_upload(m, &m.t16.tfa, ftfa)) || (rc = mixed_upload(m, &m.t16.tva, ftva)) ||
        (rc = mixed_upload(m, &m.t16.tvp, ftvp)) || (rc = mixed_upload(m, &m.t16.tfm, ftfm)) ||
        (rc = mixed_upload(m, &m.t16.tfl, ftfl)) || (rc = mixed_upload(m, &m.t16.t0, t0)) ||
        (rc = mixed_upload(m, &m.t16.mv, mv)) || (rc = mixed_upload(m, &m.t16.wf, wf)))
        return rc;
    m.nfgroups = (int)m.hfg16.size();
    m.negroups = (int)m.heg16.size();
    if ((rc = mixed_upload(m, &m.fgroups16, m.hfg16)) || (rc = mixed_upload(m, &m.egroups16, m.heg16))) return rc;
    return mixed_alloc(m, &m.rec, (size_t)nface * moment_rec_words(NB));
}

// Whether a mesh runs in groups of sixteen. One warp then holds five times the items of a group of three, so
// there must be enough groups to fill the SMs several times over: measured per step against groups of three
// (us, 6 n^3 tets), P1 86 -> 80 at n = 14 and 51 -> 63 at n = 11; P2 205 -> 202 at n = 18, 108 -> 124 at 14;
// P3 174 -> 170 at n = 14, 100 -> 125 at 11; P4 184 -> 176 at n = 11, 90 -> 174 at 8. From four groups per SM on a
// scheduler has two P4 warps: 199 -> 222 at n = 12, 228 -> 226 at n = 13, so not between. And the groups must be
// reasonably full: a mesh with many classes of face maps leaves the remainder of each class in a partial
// group, which costs as much as a full one.
inline bool wide_groups(MixedData& m, const std::vector<FaceInfo>& hfi, const std::vector<ElemFace>& hef, int64_t nowned) {
    const int64_t least = (int64_t)(m.order == 4 ? 3 : 10) * m.sms;
    if (nowned < least * kRows) return false;
    const int64_t per_sm = (int64_t)kRows * m.sms;
    if (m.order == 4 && nowned > 4 * per_sm && 2 * nowned < 11 * per_sm) return false;
    build_groups(hfi, hef, nowned, m.hfg16, m.heg16, &m.nfgroups_inner);
    if ((int64_t)m.heg16.size() * kRows * 3 <= nowned * 4 && (int64_t)m.hfg16.size() * kRows * 3 <= (int64_t)hfi.size() * 4)
        return true;
    m.hfg16.clear();
    m.heg16.clear();
    return false;
}

inline int init_mixed(MixedData& m, const Tables& tab, const std::vector<double>& hgeo,
                      const std::vector<FaceInfo>& hfi, const std::vector<ElemFace>& hef, int64_t ncell,
                      int64_t nowned, int64_t nface, double gamma, int flux, int qv, int qf, const double* d_geo,
                      const FaceInfo* d_fi, const ElemFace*, const double*) {
    if (!mixed_supported(tab.order, qv, qf)) return DG_E_ARG;
    const int NB = tab.nb, NQV = tab.nqv, NQF = tab.nqf;
    const int KB = pad8(NB - 1), MF = pad8(NQF), MV = pad8(NQV), MJ = pad8(NB), KV = pad8(3 * NQV), KF = pad8(NQF);
    m.order = tab.order; m.qv = qv; m.qf = qf; m.nb = NB; m.nqv = NQV; m.nqf = NQF;
    m.ncell = ncell; m.nface = nface; m.gamma = (float)gamma; m.flux = flux;
    m.fi = d_fi; m.geo = d_geo;
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&m.sms, cudaDevAttrMultiProcessorCount, dev);
    m.hface_cells.resize(2 * hfi.size());
    for (size_t f = 0; f < hfi.size(); ++f) {
        m.hface_cells[2 * f] = hfi[f].c0;
        m.hface_cells[2 * f + 1] = hfi[f].c1;
    }
    std::vector<double> inv_mass(NB, 0.0);
    for (int j = 0; j < NB; ++j) inv_mass[j] = 1.0 / tab.mass_ref[j];
    double wsum = 0.0;
    for (int g = 0; g < NQF; ++g) wsum += tab.w_f[g];
    m.t.wsum = wsum;
    int rc;
    if ((rc = mixed_upload(m, &m.t.inv_mass, inv_mass))) return rc;
    m.wide = wide_groups(m, hfi, hef, nowned);
    if (m.wide) {
        if ((rc = init_mixed16(m, tab, nface, qf))) return rc;
        m.ready = true;
        return DG_OK;
    }
    std::vector<double> tva(MV * KB, 0.0), tvp(MJ * KV, 0.0);
    std::vector<double> mv(NB * 3, 0.0), mf(24 * NB, 0.0), inv_detj(ncell, 0.0);
    std::vector<uint32_t> ftfa, ftva, ftvp, ftfl;
    for (int p = 0; p < 24; ++p) {
        std::vector<double> tfa(MF * KB, 0.0), tfl(MJ * KF, 0.0);
        for (int g = 0; g < NQF; ++g)
            for (int b = 1; b < NB; ++b) tfa[g * KB + (b - 1)] = tab.phi_f[((size_t)p * NQF + g) * NB + b];
        for (int j = 0; j < NB; ++j)
            for (int g = 0; g < NQF; ++g) {
                const double v = tab.w_f[g] * tab.phi_f[((size_t)p * NQF + g) * NB + j];
                tfl[j * KF + g] = v;
                mf[p * NB + j] += v;
            }
        append_frag_table(tfa, MF, KB, ftfa);
        append_frag_table(tfl, MJ, KF, ftfl);
    }
    for (int g = 0; g < NQV; ++g)
        for (int b = 1; b < NB; ++b) tva[g * KB + (b - 1)] = tab.phi_v[g * NB + b];
    for (int j = 0; j < NB; ++j)
        for (int g = 0; g < NQV; ++g)
            for (int d = 0; d < 3; ++d) {
                const double v = tab.dphi_vw[(g * NB + j) * 3 + d];
                tvp[j * KV + 3 * g + d] = v;
                mv[j * 3 + d] += v;
            }
    append_frag_table(tva, MV, KB, ftva);
    append_frag_table(tvp, MJ, KV, ftvp);
    for (int64_t e = 0; e < ncell; ++e) inv_detj[e] = 1.0 / hgeo[10 * e + 9];
    if ((rc = mixed_upload(m, &m.t.tfa, ftfa)) || (rc = mixed_upload(m, &m.t.tva, ftva)) ||
        (rc = mixed_upload(m, &m.t.tvp, ftvp)) || (rc = mixed_upload(m, &m.t.tfl, ftfl)))
        return rc;
    if ((rc = mixed_upload(m, &m.t.mv, mv)) || (rc = mixed_upload(m, &m.t.mf, mf)) ||
        (rc = mixed_upload(m, &m.t.wf32, std::vector<float>(tab.w_f.begin(), tab.w_f.end()))) ||
        (rc = mixed_upload(m, &m.inv_detj, inv_detj)))
        return rc;
    std::vector<FaceGroup> fg;
    std::vector<ElemGroup> eg;
    build_groups(hfi, hef, nowned, fg, eg, &m.nfgroups_inner);  // element groups: owned cells only
    m.nfgroups = (int)fg.size();
    m.negroups = (int)eg.size();
    if ((rc = mixed_upload(m, &m.fgroups, fg)) || (rc = mixed_upload(m, &m.egroups, eg))) return rc;
    m.hfg = fg;
    m.heg = eg;
    // padding columns of the A rows stay zero: allocation clears them and no kernel writes them
    if ((rc = mixed_alloc(m, &m.dev, (size_t)nface * face_rec_words(NQF)))) return rc;
    m.ready = true;
    return DG_OK;
}

inline void free_mixed(MixedData& m) {
    for (void* p : m.bufs) cudaFree(p);
    m.bufs.clear();
    m.ready = false;
}

inline void set_mixed_dirichlet(MixedData& m, const double* UD) { m.UD = UD; }

inline MixedFaceArgs face_args(const MixedData& m, const double* U, int face_mask, int g0 = 0, int g1 = -1) {
    MixedFaceArgs fa;
    fa.U = U; fa.fi = m.fi; fa.groups = m.fgroups; fa.UD = m.UD; fa.dev = m.dev;
    fa.t = m.t; fa.ngroups = m.nfgroups; fa.gamma = m.gamma; fa.flux = m.flux;
    if (g1 >= 0) {  // face groups [g0, g1) only
        fa.groups = m.fgroups + g0;
        fa.ngroups = g1 - g0;
    }
    fa.faces_mask = face_mask;
    return fa;
}

inline MixedElemArgs elem_args(const MixedData& m, const double* U, const double* U0, double* out, int mode,
                               double dt, double a0, double a1, int with_volume) {
    MixedElemArgs ea;
    ea.U = U; ea.U0 = U0; ea.out = out;
    ea.dev = m.dev; ea.geo = m.geo; ea.inv_detj = m.inv_detj; ea.groups = m.egroups;
    ea.t = m.t; ea.ngroups = m.negroups; ea.gamma = m.gamma; ea.volume = with_volume;
    ea.dt = dt; ea.a0 = a0; ea.a1 = a1; ea.mode = mode;
    ea.dt_inst = mode == 1 ? m.dt_inst : nullptr; ea.elem_inst = m.elem_inst;
    ea.Rv = mode == 1 ? m.Rv : nullptr;
    ea.err = m.err;
    return ea;
}

inline bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

inline Mixed16FaceArgs face_args16(const MixedData& m, const double* U, int face_mask, int g0 = 0, int g1 = -1) {
    Mixed16FaceArgs a;
    a.U = U; a.fi = m.fi; a.groups = m.fgroups16; a.UD = m.UD; a.rec = m.rec; a.t = m.t16;
    a.ngroups = m.nfgroups; a.gamma = m.gamma; a.flux = m.flux; a.faces_mask = face_mask; a.err = m.err;
    a.vec = m.nb % 2 == 0 && aligned16(U);
    if (g1 >= 0) {  // face groups [g0, g1) only
        a.groups += g0;
        a.ngroups = g1 - g0;
    }
    return a;
}

inline Mixed16ElemArgs elem_args16(const MixedData& m, const double* U, const double* U0, double* out, int mode,
                                   double dt, double a0, double a1, int with_volume) {
    Mixed16ElemArgs a;
    a.U = U; a.U0 = U0; a.out = out; a.rec = m.rec; a.geo = m.geo; a.groups = m.egroups16;
    a.t = m.t16; a.ngroups = m.negroups; a.gamma = m.gamma; a.volume = with_volume; a.dt = dt; a.a0 = a0; a.a1 = a1;
    a.mode = mode; a.dt_inst = mode == 1 ? m.dt_inst : nullptr; a.elem_inst = m.elem_inst;
    a.Rv = mode == 1 ? m.Rv : nullptr;
    a.vec = m.nb % 2 == 0 && aligned16(U) && aligned16(U0) && aligned16(out);
    a.err = m.err;
    return a;
}

// which: 0 = face fluxes, 1 = element kernel (volume + face integrals + update).
template <int NB, int NQV, int NQF, int WE>
inline int mixed_launch(MixedData& m, int which, const double* U, const double* U0, double* out, int mode,
                        double dt, double a0, double a1, int face_mask, int with_volume, cudaStream_t s, int g0,
                        int g1) {
    if (which == 0) {
        constexpr int W = 4;  // 4-warp CTAs: finer-grained scheduling than 8 at the same occupancy
        const int n = g1 < 0 ? m.nfgroups : g1 - g0;
        const int g = (int)std::min<int64_t>((n + W - 1) / W, (int64_t)m.sms * 64);
        return launch_early(face_flux_mixed<NB, NQF, W>, g, W * 32, 0, s, face_args(m, U, face_mask, g0, g1));
    } else if (m.elem_kernel == 2 && (5 * NB * 8) % 16 == 0 && ((uintptr_t)U & 15) == 0 &&
               ((uintptr_t)U0 & 15) == 0) {
        if constexpr ((5 * NB * 8) % 16 == 0) {
            const auto ea = elem_args(m, U, U0, out, mode, dt, a0, a1, with_volume);
            if (m.elem_ctas == 2) {
                constexpr int W = elem_staged_warps<NB, NQV, NQF>(2);
                constexpr size_t smem = elem_staged_warp_smem<NB, NQV, NQF>() * W;
                static unsigned long long done = 0;
                int rc = ensure_smem(element_mixed_staged<NB, NQV, NQF, W, 2>, smem, done);
                if (rc) return rc;
                const int g = (int)std::min<int64_t>((m.negroups + W - 1) / W, (int64_t)m.sms * 2);
                return launch_early(element_mixed_staged<NB, NQV, NQF, W, 2>, g, W * 32, smem, s, ea);
            } else {
                constexpr int W = elem_staged_warps<NB, NQV, NQF>(1);
                constexpr size_t smem = elem_staged_warp_smem<NB, NQV, NQF>() * W;
                static unsigned long long done = 0;
                int rc = ensure_smem(element_mixed_staged<NB, NQV, NQF, W, 1>, smem, done);
                if (rc) return rc;
                const int g = (int)std::min<int64_t>((m.negroups + W - 1) / W, (int64_t)m.sms);
                return launch_early(element_mixed_staged<NB, NQV, NQF, W, 1>, g, W * 32, smem, s, ea);
            }
        }
    } else {
        constexpr size_t smem = sizeof(ElemMixedSmem<NB, NQV, NQF>) * WE;
        static unsigned long long done = 0;
        int rc = ensure_smem(element_mixed<NB, NQV, NQF, WE>, smem, done);
        if (rc) return rc;
        const int g = (int)std::min<int64_t>((m.negroups + WE - 1) / WE, (int64_t)m.sms * 32);
        return launch_early(element_mixed<NB, NQV, NQF, WE>, g, WE * 32, smem, s,
                            elem_args(m, U, U0, out, mode, dt, a0, a1, with_volume));
    }
    return DG_E_ARG;  // staged, of a row length that excludes it: not reached
}

// Element-kernel shapes of the two-launch schedule that dg_autotune times: the kernel (0: loads
// phase by phase, 2: rows staged by bulk copies), warps per CTA (three elements each) and resident
// CTAs per SM. Returns how many apply to this order and rule pair.
struct ElemShape {
    int kernel, warps, ctas, group = 3;  // items per warp
};
inline int mixed_elem_shapes(const MixedData& m, ElemShape out[3]) {
    if (m.wide) {  // groups of sixteen: one shape, its rows always staged
        out[0] = ElemShape{2, mixed16_element_warps(m.order, m.qv, m.qf), 1, kRows};
        return 1;
    }
#define X(P, QV, QF, NB, NQV, NQF, W)                                                 \
    if (m.order == P && m.qv == QV && m.qf == QF) {                                   \
        int n = 0;                                                                    \
        out[n++] = ElemShape{0, W, W == 8 ? 3 : 6};                                   \
        if ((5 * NB * 8) % 16 == 0) {                                                 \
            out[n++] = ElemShape{2, elem_staged_warps<NB, NQV, NQF>(1), 1};           \
            out[n++] = ElemShape{2, elem_staged_warps<NB, NQV, NQF>(2), 2};           \
        }                                                                             \
        return n;                                                                     \
    }
    FVEDG_MIXED_COMBOS(X)
#undef X
    return 0;
}

// Face launches (which 0) cover face groups [g0, g1) (g1 < 0: all of them).
inline int mixed_kernel(MixedData& m, int which, const double* U, const double* U0, double* out, int mode,
                        double dt, double a0, double a1, int face_mask, int with_volume, cudaStream_t s,
                        std::atomic<int64_t>* launches, int g0 = 0, int g1 = -1) {
    if (!m.ready) return DG_E_ARG;
    if (which == 0 && g1 >= 0 && g1 <= g0) return DG_OK;  // an empty range: nothing to launch
    ++*launches;
    if (m.wide)
        return which == 0 ? mixed16_face(m.order, m.qv, m.qf, m.sms, face_args16(m, U, face_mask, g0, g1), s)
                          : mixed16_element(m.order, m.qv, m.qf, m.sms,
                                            elem_args16(m, U, U0, out, mode, dt, a0, a1, with_volume), s);
#define X(P, QV, QF, NB, NQV, NQF, W)                                                                           \
    if (m.order == P && m.qv == QV && m.qf == QF)                                                               \
        return mixed_launch<NB, NQV, NQF, W>(m, which, U, U0, out, mode, dt, a0, a1, face_mask, with_volume, s, \
                                             g0, g1);
    FVEDG_MIXED_COMBOS(X)
#undef X
    return DG_E_ARG;
}

// One stage: face fluxes, then the element kernel.
template <class Timed>
inline int mixed_stage(MixedData& m, const double* U, const double* U0, double* out, int mode, double dt, double a0,
                       double a1, int face_mask, int with_volume, cudaStream_t s, std::atomic<int64_t>* launches,
                       Timed&& timed) {
    auto K = [&](int which) {
        return mixed_kernel(m, which, U, U0, out, mode, dt, a0, a1, face_mask, with_volume, s, launches);
    };
    const int rc = timed(0, [&] { return K(0); });
    if (rc) return rc;
    return timed(1, [&] { return K(1); });
}

inline int residual_mixed(MixedData& m, const double* U, double* R, int part, cudaStream_t s,
                          std::atomic<int64_t>* launches) {
    const int mask = part == 0 ? 3 : part == 1 ? 0 : part == 2 ? 1 : 2;
    return mixed_stage(m, U, U, R, 0, 0.0, 0.0, 0.0, mask, part == 0 || part == 1, s, launches,
                       [](int, auto&& fn) { return fn(); });
}

inline int mixed_launches_per_step(const MixedData&) { return 6; }

// SSP-RK3 step; `timed(cls, fn)` runs fn (one launch) and may bracket it with timing events.
// `post(in, out, st)` runs after every stage st (the limiter, or nothing). Stages st0..st1-1 only
// (one stage at a time when a halo exchange runs between stages).
template <class Timed, class Post>
inline int step_mixed(MixedData& m, double* Un, double* Ua, double* Ub, double dt, cudaStream_t s,
                      std::atomic<int64_t>* launches, Timed&& timed, Post&& post, int st0 = 0, int st1 = 3) {
    const double A0[3] = {0.0, 0.75, 1.0 / 3.0};
    const double A1[3] = {1.0, 0.25, 2.0 / 3.0};
    const double* in[3] = {Un, Ua, Ub};
    double* out[3] = {Ua, Ub, Un};
    for (int st = st0; st < st1; ++st) {
        int rc = mixed_stage(m, in[st], Un, out[st], 1, dt, A0[st], A1[st], 3, 1, s, launches, timed);
        if (rc || (rc = post(in[st], out[st], st))) return rc;
    }
    return DG_OK;
}

}  // namespace fvedg
