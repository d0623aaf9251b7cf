"""What a context keeps between calls for speed alone (build scratch, the raster's
lists, a finished column plan) goes back before an allocation is refused."""
import os
import shutil
import subprocess

import pytest


def test_failed_allocations_give_back_kept_memory(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if shutil.which("g++") is None or not os.path.exists(os.path.join(include, "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers not available")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    exe = tmp_path / "spare_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wno-deprecated-declarations", "-I", include,
                    os.path.join(root, "tests", "cpp", "spare_check.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and "spare memory ok" in r.stdout, r.stdout + r.stderr
