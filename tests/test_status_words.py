"""What a call reports of its bounded waits (dg_status_words.h): a context's words and the tile queue's error, both taken and
cleared by the call that reports them."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
CXX = shutil.which("g++")

PROGRAM = r"""
#include <cstdio>
#include "dg_status_words.h"
using namespace fvedg;
extern "C" cudaError_t cudaHostAlloc(void**, size_t, unsigned) { return cudaErrorMemoryAllocation; }
int main() {
    for (int word = -1; word < kStatusWords; ++word)
        for (int queue = 0; queue < 2; ++queue) {
            int words[kStatusWords] = {}, error = queue ? DG_E_WATCHDOG : DG_OK, cleared = 0;
            if (word >= 0) words[word] = DG_E_WATCHDOG;
            auto call = [&] {
                return take_status(words, [&](int* e) { *e = error; return (int)DG_OK; },
                                   [&] { ++cleared; error = DG_OK; return (int)DG_OK; });
            };
            const int first = call(), second = call();
            if (first != (word >= 0 || queue ? DG_E_WATCHDOG : DG_OK) || second != DG_OK || cleared != queue) {
                std::printf("word %d queue %d: %d, then %d\n", word, queue, first, second);
                return 1;
            }
        }
    int words[kStatusWords] = {};
    auto none = [](int*) { return (int)DG_OK; };
    if (take_status(words, [](int*) { return (int)DG_E_CUDA; }, [] { return (int)DG_OK; }) != DG_E_CUDA) return 2;
    if (take_status(words, [](int* e) { *e = DG_E_WATCHDOG; return (int)DG_OK; }, [] { return (int)DG_E_CUDA; }) != DG_E_CUDA) return 3;
    return take_status(words, none, [] { return (int)DG_OK; }) == DG_OK && take_status(words) == DG_OK ? 0 : 4;
}
"""


@pytest.mark.skipif(CXX is None or not os.path.isdir(CUDA), reason="needs a C++ compiler and the CUDA headers")
def test_a_call_takes_all_it_reports(tmp_path):
    (tmp_path / "main.cpp").write_text(PROGRAM)
    exe = str(tmp_path / "main")
    subprocess.run([CXX, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "include"), "-I", os.path.join(CUDA, "include"),
                    "-I", os.path.join(ROOT, "fve_dg_b200", "csrc"), str(tmp_path / "main.cpp"), "-o", exe], check=True)
    done = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert done.returncode == 0, done.stdout
