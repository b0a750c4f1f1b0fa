"""The groups of items with equal face maps (dg_groups.h) against their definition in an ordered map: few and many
classes, ghost cells, partial groups, and a number of items that is no multiple of the group."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CXX = shutil.which("g++")

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include <map>
#include <random>
#include "dg_groups.h"
using namespace fvedg;
namespace fvedg {
const int kPermSlots[kNumPerms][3] = {{0,1,2},{0,1,3},{0,2,1},{0,2,3},{0,3,1},{0,3,2},{1,0,2},{1,0,3},{1,2,0},{1,2,3},{1,3,0},{1,3,2},
                                      {2,0,1},{2,0,3},{2,1,0},{2,1,3},{2,3,0},{2,3,1},{3,0,1},{3,0,2},{3,1,0},{3,1,2},{3,2,0},{3,2,1}};
}
struct Face { int c0, c1, meta; };
struct Elem { int face, meta; };
template <int N> struct FaceN { int f[N]; int n; };
template <int N> struct ElemN { int e[N]; int face[N][4]; int meta[4]; int n; };

template <int N>
static bool check(const std::vector<Face>& hf, const std::vector<Elem>& he, int64_t ncell) {
    std::vector<FaceN<N>> fg, want_f;
    std::vector<ElemN<N>> eg, want_e;
    int inner = -1, want_inner = -1;
    build_groups(hf, he, ncell, fg, eg, &inner);
    for (int halo = 0; halo < 2; ++halo) {
        std::map<int64_t, FaceN<N>> open;
        for (size_t f = 0; f < hf.size(); ++f) {
            if ((hf[f].c0 >= ncell || hf[f].c1 >= ncell) != (halo == 1)) continue;
            FaceN<N>& g = open[(int64_t)(hf[f].meta & 0xffffff) * 2 + (hf[f].c1 >= 0)];
            g.f[g.n++] = (int)f;
            if (g.n == N) { want_f.push_back(g); g = FaceN<N>{}; }
        }
        for (auto& kv : open)
            if (kv.second.n) {
                for (int i = kv.second.n; i < N; ++i) kv.second.f[i] = kv.second.f[0];
                want_f.push_back(kv.second);
            }
        if (!halo) want_inner = (int)want_f.size();
    }
    std::map<int64_t, ElemN<N>> open;
    for (int64_t e = 0; e < ncell; ++e) {
        int face[4], meta[4];
        int64_t key = 0;
        for (int i = 0; i < 4; ++i) {
            const int* s = kPermSlots[he[4 * e + i].meta & 0xff];
            face[6 - s[0] - s[1] - s[2]] = he[4 * e + i].face;
            meta[6 - s[0] - s[1] - s[2]] = he[4 * e + i].meta;
        }
        for (int q = 0; q < 4; ++q) key = key * 65536 + meta[q];
        ElemN<N>& g = open[key];
        g.e[g.n] = (int)e;
        for (int q = 0; q < 4; ++q) { g.face[g.n][q] = face[q]; g.meta[q] = meta[q]; }
        if (++g.n == N) { want_e.push_back(g); g = ElemN<N>{}; }
    }
    for (auto& kv : open)
        if (ElemN<N> g = kv.second; g.n) {
            for (int i = g.n; i < N; ++i) {
                g.e[i] = g.e[0];
                for (int q = 0; q < 4; ++q) g.face[i][q] = g.face[0][q];
            }
            want_e.push_back(g);
        }
    return inner == want_inner && fg.size() == want_f.size() && eg.size() == want_e.size() &&
           !std::memcmp(fg.data(), want_f.data(), fg.size() * sizeof(fg[0])) &&
           !std::memcmp(eg.data(), want_e.data(), eg.size() * sizeof(eg[0]));
}

int main() {
    std::mt19937 r(7);
    for (int maps : {1, 3, 24})
        for (int64_t ncell : {1, 5, 1000, 5003})
            for (int ghosts : {0, 37}) {
                const int64_t all = ncell + ghosts;
                std::vector<Face> hf(2 * ncell + 1);
                for (Face& f : hf) {
                    f.c0 = (int)(r() % all);
                    f.c1 = r() % 9 ? (int)(r() % all) : -1;
                    f.meta = (int)(r() % maps) | (int)(r() % maps) << 8 | (int)(r() % 2 * 5) << 16 | (int)(r() % 2) << 24;
                }
                std::vector<Elem> he(4 * all);
                for (int64_t e = 0; e < all; ++e)
                    for (int i = 0; i < 4; ++i)  // any of the maps whose face lies opposite vertex (i + turn) % 4
                        for (int p = (int)(r() % 24), turn = maps > 3 ? (int)(e % 4) : 0;; p = (p + 1) % 24)
                            if (6 - kPermSlots[p][0] - kPermSlots[p][1] - kPermSlots[p][2] == (i + turn) % 4) {
                                he[4 * e + i] = Elem{(int)(r() % hf.size()), (maps == 1 ? p / 6 * 6 : p) | (int)(r() % 2) << 8};
                                if (maps == 1)
                                    for (int k = 0; k < 24; ++k)
                                        if (6 - kPermSlots[k][0] - kPermSlots[k][1] - kPermSlots[k][2] == (i + turn) % 4) {
                                            he[4 * e + i].meta = k;
                                            break;
                                        }
                                break;
                            }
                if (!check<3>(hf, he, ncell) || !check<8>(hf, he, ncell) || !check<16>(hf, he, ncell)) {
                    std::printf("maps %d cells %ld ghosts %d\n", maps, (long)ncell, ghosts);
                    return 1;
                }
            }
    return 0;
}
"""


@pytest.mark.skipif(CXX is None, reason="needs g++")
def test_groups(tmp_path):
    src, exe = tmp_path / "groups.cpp", tmp_path / "groups"
    src.write_text(PROGRAM)
    subprocess.run([CXX, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "fve_dg_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
                    str(src), "-o", str(exe)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stdout
