"""A host allocation that fails within a call on a batch of uneven orders leaves the
context as it was (tests/cpp/test_exceptions.cpp, built against the library)."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_failed_host_allocations(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    from zest_gb300 import build
    build.build()
    exe, lib = str(tmp_path / "test_exceptions"), os.path.join(ROOT, "zest_gb300")
    res = subprocess.run([nvcc, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "include"),
                          os.path.join(ROOT, "tests", "cpp", "test_exceptions.cpp"), "-L", lib, "-lzest_gb300",
                          "-Xlinker", "-rpath", "-Xlinker", lib, "-o", exe], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    res = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout + res.stderr
    ok, thrown = res.stdout.split()
    assert ok == "ok" and int(thrown) > 4  # work lists, tile lists and GEMM units of both precisions
