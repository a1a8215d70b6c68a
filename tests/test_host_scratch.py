"""Page-locked scratch of a call that is left by an exception
(single-svdlib_b200/csrc/host_scratch.h), compiled with g++ against a fake
stream: the copies in flight end before the pool may hand it on."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "single-svdlib_b200", "csrc")
CUDA_INC = "/usr/local/cuda/include"
MAIN = r"""
#include <cstdio>
#include <stdexcept>
#include "host_scratch.h"
static int in_flight = 0, out = 0;
static cudaStream_t mine = (cudaStream_t)0x10;
cudaError_t CUDARTAPI cudaStreamSynchronize(cudaStream_t s) { if (s == mine) in_flight = 0; return cudaSuccess; }
namespace svdb {
void* host_result_alloc(size_t n) { ++out; return new char[n]; }
void host_result_free(void* p) {
    if (in_flight) { std::printf("handed back under a copy\n"); throw 1; }
    --out;
    delete[] (char*)p;
}
}
int main() {
    try {
        svdb::HostScratch h(64 << 10, mine);
        in_flight = 1;  // a copy into it
        throw std::runtime_error("a product failed");
    } catch (std::runtime_error&) {
    }
    std::printf("%d %d\n", in_flight, out);
}
"""


def test_scratch_waits_for_its_copies(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None or not os.path.exists(os.path.join(CUDA_INC, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    (tmp_path / "m.cpp").write_text(MAIN)
    exe = str(tmp_path / "m")
    subprocess.run([cxx, "-O1", "-std=c++17", "-I", CSRC, "-I", CUDA_INC, str(tmp_path / "m.cpp"), "-o", exe], check=True)
    res = subprocess.run([exe], capture_output=True, text=True)
    assert res.returncode == 0 and res.stdout == "0 0\n", res.stdout + res.stderr
