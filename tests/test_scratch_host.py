"""Host logic of the scratch pool and the mapped host words, against a fake CUDA runtime (no GPU)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_scratch_host_logic(tmp_path):
    from morpheus_gb300 import build as B
    if shutil.which(B.NVCC) is None:
        pytest.skip("needs nvcc")
    obj, exe = str(tmp_path / "scratch.o"), str(tmp_path / "test_scratch_host")
    r = subprocess.run([B.NVCC, *B.NVCC_FLAGS, "-c", os.path.join(B.CSRC, "scratch.cu"), "-o", obj],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(shutil.which(B.NVCC)))), "include")
    r = subprocess.run(["g++", "-std=c++17", "-I", include, "-I", B.INCLUDE, "-I", B.CSRC,
                        os.path.join(ROOT, "tests", "cpp", "test_scratch_host.cpp"), obj, "-o", exe, "-lpthread"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
