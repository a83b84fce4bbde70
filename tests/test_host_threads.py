"""The library's host state under several threads (CPU only).

libcuopus.cu is compiled as it is and linked with a CUDA runtime made for the
test (tests/fake_cuda_driver.cpp), under ThreadSanitizer: a server's thread
resamples on one device while a program's calls decode and resample on another."""
import os
import shutil
import subprocess

import pytest

from cuopus_b200.build import ARCH, CSRC, NVCC

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_resampler_shares_no_unlocked_state(tmp_path):
    if not os.path.exists(NVCC) or not shutil.which("g++"):
        pytest.skip("nvcc and g++ are needed")
    inc = os.path.join(os.path.dirname(os.path.dirname(NVCC)), "include")
    lib, exe = str(tmp_path / "libcuopus.o"), str(tmp_path / "threads")
    subprocess.run([NVCC, *ARCH, "-O1", "-std=c++17", "-Xcompiler", "-fsanitize=thread,-g", "-I", CSRC, "-cudart", "none",
                    "-c", os.path.join(CSRC, "libcuopus.cu"), "-o", lib], check=True, capture_output=True)
    subprocess.run(["g++", "-O1", "-g", "-std=c++17", "-w", "-fsanitize=thread", "-I", inc, "-c",
                    os.path.join(ROOT, "tests", "fake_cuda_driver.cpp"), "-o", exe + ".o"], check=True, capture_output=True)
    # what these threads never call (demuxing, graphs, events) stays unresolved
    subprocess.run(["g++", "-fsanitize=thread", exe + ".o", lib, "-o", exe, "-lpthread",
                    "-Wl,--unresolved-symbols=ignore-all"], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, TSAN_OPTIONS="halt_on_error=0:exitcode=66"))
    assert r.returncode == 0, (r.stdout + r.stderr)[-4000:]
