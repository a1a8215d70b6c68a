"""Which operators the resident Lanczos cluster takes
(single-svdlib_b200/csrc/lz_resident.h), compiled with g++ into
tests/lz_resident_check.cpp."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "single-svdlib_b200", "csrc")
CUDA_INC = "/usr/local/cuda/include"


def test_resident_choice(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None or not os.path.exists(os.path.join(CUDA_INC, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path / "lz_resident_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", CSRC, "-I", CUDA_INC,
                    os.path.join(ROOT, "tests", "lz_resident_check.cpp"), "-o", exe], check=True)
    res = subprocess.run([exe], capture_output=True, text=True)
    assert res.returncode == 0 and res.stdout == "ok\n", res.stdout + res.stderr
