"""The staging of host arrays (dg_transfer.cuh) on a stand-in for the CUDA runtime: several transfers at once make no
more than two pinned blocks and make them once, and a call at the heap's limit copies all the same and throws nothing."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
CXX = shutil.which("g++")

PROGRAM = r"""
#include <cuda_runtime.h>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <thread>
#include <vector>

static std::atomic<int> allocs{0}, live{0}, inside{0};
static int together = 1;
static thread_local bool no_heap = false;
void* operator new(size_t n) {
    void* p = no_heap ? nullptr : std::malloc(n);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

extern "C" {
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { ++allocs; ++live; *p = std::malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { --live; std::free(p); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)std::malloc(1); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free((void*)e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { a->type = cudaMemoryTypeUnregistered; return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
}
#include "dg_transfer.cuh"
using namespace fvedg;

static const size_t kBlk = 400;
static const int64_t kRow = 12000;  // 4.8 MB

// One transfer in and out, packed or apart; 1 where the pool had no block for it.
static int copy(size_t stride) {
    std::vector<char> host(kRow * stride, 1), dev(kRow * kBlk, 0);
    for (int64_t i = 0; i < kRow; ++i)
        for (size_t k = 0; k < kBlk; ++k) host[i * stride + k] = (char)(i * 7 + k);
    const std::vector<char> was = host;
    no_heap = together == 1;
    int rc = staged_copy(true, dev.data(), host.data(), stride, kBlk, kRow, 0, nullptr);
    no_heap = false;
    if (rc) return rc;
    for (int64_t i = 0; i < kRow; ++i)
        if (std::memcmp(&dev[i * kBlk], &was[i * stride], kBlk)) std::abort();
    std::fill(host.begin(), host.end(), 1);
    no_heap = together == 1;
    rc = staged_copy(false, dev.data(), host.data(), stride, kBlk, kRow, 0, nullptr);
    no_heap = false;
    if (rc) return rc;
    if (host != was) std::abort();
    return 0;
}

int main() {
    { StageUse first; if (copy(kBlk)) return 1; }
    if (live) return 2;  // none once the last context is gone
    {
        StageUse use;
        if (copy(kBlk) || copy(kBlk + 24)) return 3;  // at the heap's limit
        together = 5;
        allocs = 1;
        std::vector<std::thread> t;
        std::atomic<int> ready{0}, taken{0};
        for (int i = 0; i < together; ++i)
            t.emplace_back([&] {
                ++ready;
                while (ready < together) std::this_thread::yield();
                for (int k = 0; k < 20; ++k) {
                    const int rc = copy(kBlk);
                    if (rc == 0) ++taken;
                    else if (rc != 1) std::abort();
                }
            });
        for (auto& x : t) x.join();
        if (taken < 2 || allocs > 2 || live > 2) { std::printf("%d blocks made, %d there\n", (int)allocs, (int)live); return 4; }
    }
    return live ? 5 : 0;
}
"""


@pytest.mark.skipif(CXX is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")), reason="needs g++ and the CUDA headers")
def test_pool(tmp_path):
    src, exe = tmp_path / "pool.cpp", tmp_path / "pool"
    src.write_text(PROGRAM)
    csrc = os.path.join(ROOT, "fve_dg_b200", "csrc")
    subprocess.run([CXX, "-std=c++17", "-O1", "-pthread", "-I", csrc, "-I", os.path.join(ROOT, "include"), "-I", os.path.join(CUDA, "include"),
                    str(src), "-o", str(exe)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, (run.returncode, run.stdout, run.stderr)
