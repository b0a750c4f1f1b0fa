// Groups of items whose face maps are equal, host side: the kernels take a group of N faces or elements at a time.
#pragma once
#include <algorithm>
#include <cstdint>
#include <vector>

#include "dg_internal.h"

namespace fvedg {

// Small integers for keys as they come, by open addressing; far cheaper here than an ordered map's search per item.
class KeyIndex {
  public:
    explicit KeyIndex(int bits = 8) : bits_(bits), at_((size_t)1 << bits, -1) {}
    // The number of `key`, counted from 0; `keys()[n]` is key number n.
    int of(int64_t key) {
        if (last_ >= 0 && keys_[last_] == key) return last_;
        size_t h = slot(key);
        while (at_[h] >= 0 && keys_[at_[h]] != key) h = (h + 1) & (at_.size() - 1);
        if (at_[h] < 0) {
            at_[h] = (int)keys_.size();
            keys_.push_back(key);
            if (2 * keys_.size() > at_.size()) grow();
            return last_ = (int)keys_.size() - 1;
        }
        return last_ = at_[h];
    }
    const std::vector<int64_t>& keys() const { return keys_; }

  private:
    size_t slot(int64_t key) const { return (size_t)(((uint64_t)key * 0x9E3779B97F4A7C15ull) >> (64 - bits_)); }
    void grow() {
        at_.assign((size_t)1 << ++bits_, -1);
        for (size_t i = 0; i < keys_.size(); ++i) {
            size_t h = slot(keys_[i]);
            while (at_[h] >= 0) h = (h + 1) & (at_.size() - 1);
            at_[h] = (int)i;
        }
    }
    int bits_, last_ = -1;
    std::vector<int> at_;
    std::vector<int64_t> keys_;
};

// The order of the keys, for the groups that are left partial.
inline std::vector<int> by_key(const std::vector<int64_t>& keys) {
    std::vector<int> order(keys.size());
    for (size_t i = 0; i < order.size(); ++i) order[i] = (int)i;
    std::sort(order.begin(), order.end(), [&](int a, int b) { return keys[a] < keys[b]; });
    return order;
}

// Faces with equal (perm0, perm1, kind) and elements with equal face maps (in canonical face
// order: local face q is the one opposite local vertex q) are grouped in mesh order, N to a group. A partial group
// repeats its first member in the unused slots (never read as a row: rows of unused slots are masked by the group size).
// Face groups: first the faces between owned elements, then (from *nf_inner on) the faces touching a ghost element
// (cells >= ncell), whose fluxes need the ghost rows of a halo exchange. Element groups: the owned elements [0, ncell).
template <class FaceInfo, class ElemFace, class FG, class EG>
inline void build_groups(const std::vector<FaceInfo>& hfi, const std::vector<ElemFace>& hef, int64_t ncell,
                         std::vector<FG>& fg, std::vector<EG>& eg, int* nf_inner) {
    constexpr int N = sizeof(FG{}.f) / sizeof(int);
    fg.reserve(hfi.size() / N + 64);
    eg.reserve((size_t)ncell / N + 64);
    bool ghosts = false;
    for (int halo = 0; halo < 1 + ghosts; ++halo) {
        KeyIndex index;
        std::vector<FG> open;
        for (int64_t f = 0; f < (int64_t)hfi.size(); ++f) {
            const FaceInfo& F = hfi[f];
            const bool touches = F.c0 >= ncell || F.c1 >= ncell;
            ghosts = ghosts || touches;
            if (touches != (halo == 1)) continue;
            const int k = index.of((int64_t)(F.meta & 0xffffff) * 2 + (F.c1 >= 0 ? 1 : 0));
            if (k == (int)open.size()) open.emplace_back();
            FG& g = open[k];
            g.f[g.n++] = (int)f;
            if (g.n == N) {
                fg.push_back(g);
                g = FG{};
            }
        }
        for (int k : by_key(index.keys())) {
            FG& g = open[k];
            if (g.n == 0) continue;
            for (int i = g.n; i < N; ++i) g.f[i] = g.f[0];
            fg.push_back(g);
        }
        if (halo == 0) *nf_inner = (int)fg.size();
    }
    KeyIndex index;  // by the four face maps and sides
    std::vector<EG> open;
    for (int64_t e = 0; e < ncell; ++e) {
        int face[4] = {-1, -1, -1, -1}, meta[4] = {0, 0, 0, 0};
        for (int i = 0; i < 4; ++i) {
            const ElemFace& ef = hef[4 * e + i];
            const int p = ef.meta & 0xff;
            const int q = 6 - kPermSlots[p][0] - kPermSlots[p][1] - kPermSlots[p][2];  // missing vertex
            face[q] = ef.face;
            meta[q] = ef.meta;
        }
        int64_t key = 0;
        for (int q = 0; q < 4; ++q) key = key * 65536 + meta[q];
        const int k = index.of(key);
        if (k == (int)open.size()) open.emplace_back();
        EG& g = open[k];
        g.e[g.n] = (int)e;
        for (int q = 0; q < 4; ++q) {
            g.face[g.n][q] = face[q];
            g.meta[q] = meta[q];
        }
        if (++g.n == N) {
            eg.push_back(g);
            g = EG{};
        }
    }
    for (int k : by_key(index.keys())) {
        EG& g = open[k];
        if (g.n == 0) continue;
        for (int i = g.n; i < N; ++i) {
            g.e[i] = g.e[0];
            for (int q = 0; q < 4; ++q) g.face[i][q] = g.face[0][q];
        }
        eg.push_back(g);
    }
}

}  // namespace fvedg
