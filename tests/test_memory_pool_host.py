"""The kept device memory's bookkeeping with two devices, on the host: a program of
mem_pool.cpp and a counting stand-in for the CUDA runtime."""
import os
import subprocess

import pytest

from leo2d_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA_INCLUDE = os.path.join(build._cuda_home(), "include")


@pytest.mark.skipif(not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime_api.h")), reason="no CUDA headers")
def test_two_devices(tmp_path):
    exe = str(tmp_path / "pool")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + build.REPO, "-I" + CUDA_INCLUDE,
                    os.path.join(HERE, "memory_pool_host.cpp"), os.path.join(build.HOST, "mem_pool.cpp"), "-o", exe,
                    "-lpthread"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
