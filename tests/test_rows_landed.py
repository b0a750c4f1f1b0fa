"""A warp's bounded wait for its rows (dg_slots.cuh), with 32 threads for the lanes and a stand-in for the barrier: an
expired wait that only some lanes see, the others' last poll having found the rows, is recorded and ends for all alike."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CXX = shutil.which("g++")

STAND_IN = r"""
#pragma once
#include <cstdint>
#define __device__
#define __forceinline__ inline
namespace fvedg {
constexpr long long kBulkSpinLimit = 4;
bool mbar_wait_bounded(uint64_t* bar, unsigned parity, long long limit);
inline void mbar_arrive_expect_tx(uint64_t*, unsigned) {}
inline void mbar_expect_tx(uint64_t*, unsigned) {}
inline void mbar_arrive(uint64_t*) {}
inline void bulk_copy_g2s(void*, const void*, unsigned, uint64_t*) {}
inline uint32_t smem_addr(const void*) { return 0; }
}
bool __all_sync(unsigned, bool);
"""

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <pthread.h>
#include <thread>
#include <vector>
#include "dg_slots.cuh"
using namespace fvedg;
static pthread_barrier_t meet;
static std::atomic<int> no{0};
static thread_local bool late = false;
static thread_local int waits = 0;
bool __all_sync(unsigned, bool v) {
    if (!v) ++no;
    pthread_barrier_wait(&meet);
    const bool all = no == 0;
    pthread_barrier_wait(&meet);
    return all;
}
namespace fvedg {
bool mbar_wait_bounded(uint64_t*, unsigned, long long) { return ++waits > 1 || !late; }
}
template <bool VOTE_FIRST>
int check() {
    // which lanes are late: none, one that is not lane 0, lane 0, all but lane 0, all
    const unsigned cases[] = {0u, 1u << 5, 1u, ~1u, ~0u};
    for (unsigned mask : cases) {
        no = 0;
        int err = DG_OK;
        bool ok[32];
        int waited[32];
        unsigned parity[32] = {};
        pthread_barrier_init(&meet, nullptr, 32);
        std::vector<std::thread> warp;
        for (int lane = 0; lane < 32; ++lane)
            warp.emplace_back([&, lane] {
                static uint64_t bar;
                late = (mask >> lane) & 1;
                ok[lane] = rows_landed<VOTE_FIRST>(bar, parity[lane], &err);
                waited[lane] = waits;
            });
        for (auto& t : warp) t.join();
        pthread_barrier_destroy(&meet);
        for (int lane = 0; lane < 32; ++lane)
            if (ok[lane] != (mask == 0) || parity[lane] != 1u || waited[lane] != ((VOTE_FIRST ? mask : (mask >> lane) & 1) ? 2 : 1)) {
                std::printf("mask %x lane %d: %d, %d waits\n", mask, lane, ok[lane], waited[lane]);
                return 1;
            }
        if (err != (mask ? DG_E_WATCHDOG : DG_OK)) { std::printf("mask %x: status %d\n", mask, err); return 2; }
    }
    return 0;
}
int main() { const int rc = check<false>(); return rc ? rc : check<true>(); }
"""


@pytest.mark.skipif(CXX is None, reason="needs a C++ compiler")
def test_an_expired_wait_ends_for_the_whole_warp(tmp_path):
    shutil.copy(os.path.join(ROOT, "fve_dg_b200", "csrc", "dg_slots.cuh"), tmp_path / "dg_slots.cuh")
    (tmp_path / "dg_tma.cuh").write_text(STAND_IN)
    (tmp_path / "main.cpp").write_text(PROGRAM)
    exe = str(tmp_path / "main")
    subprocess.run([CXX, "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "include"), str(tmp_path / "main.cpp"), "-o", exe],
                   check=True)
    done = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert done.returncode == 0, done.stdout
