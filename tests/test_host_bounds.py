"""Bounds of the host-side sizing in libtuna_gpu.so (tests/cpp/host_bounds_check.cu, linked
against the library, run without a GPU)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_host_bounds(tmp_path):
    import tuna_gb300.build as B
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    lib = B.gpu_lib()
    exe = str(tmp_path / "host_bounds_check")
    src = os.path.join(ROOT, "tests", "cpp", "host_bounds_check.cu")
    r = subprocess.run([nvcc, *B.ARCH, "-std=c++17", "-O2", "--expt-relaxed-constexpr",
                        "-I", os.path.join(ROOT, "tuna_gb300", "csrc"), "-I", os.path.join(ROOT, "include"),
                        src, "-o", exe, "-L", os.path.dirname(lib), "-ltuna_gpu",
                        "-Xlinker", "-rpath," + os.path.dirname(lib)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("OK"), r.stdout + r.stderr
