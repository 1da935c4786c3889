"""Rejected kernel launches, on the host: the library against a CUDA runtime that refuses chosen launches.

tests/native/launch_failure_test.cu runs it without a GPU (fake_cuda_runtime.cpp) and checks what a rejected launch leaves
behind: no entry in the next frame's fallback list, and no error for the next call to report.
"""
import os
import shutil
import subprocess

import pytest

import tron_grid_gb300  # noqa: F401  (the package's build module lives beside it)

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "tron-grid_gb300")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    import __graft_entry__

    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    __graft_entry__.build()
    lib, native = os.path.join(PKG, "lib"), os.path.join(ROOT, "tests", "native")
    exe = tmp_path_factory.mktemp("native") / "launch_failure_test"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O1", "-cudart", "shared",
                    "-I", os.path.join(PKG, "csrc"), "-I", os.path.join(ROOT, "include"),
                    os.path.join(native, "launch_failure_test.cu"), os.path.join(native, "fake_cuda_runtime.cpp"), "-o", str(exe), "-L", lib,
                    "-ltg_svgf", "-Xlinker", "-rpath", "-Xlinker", lib, "-Xlinker", "--export-dynamic"], check=True)
    return str(exe)


@pytest.mark.parametrize("which", ["counter", "last"])
def test_rejected_launch(program, which):
    r = subprocess.run([program, which], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
