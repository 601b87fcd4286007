"""The plan of the decode GEMV and where its prepared activation lies in shared memory, on the host: every format, row count
and width."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_plan_and_layout_of_every_shape(tmp_path):
    from kraken_b200 import build
    try:
        nvcc = build.nvcc()
    except RuntimeError:
        pytest.skip("no nvcc")
    lib_dir = os.path.join(ROOT, "kraken_b200")
    if not os.path.exists(os.path.join(lib_dir, "libkrk_cuda.so")):
        build.build()
    exe = str(tmp_path / "gemv_plan")
    subprocess.run([nvcc, *build.ARCH, "-O1", "-std=c++17", "--expt-relaxed-constexpr", "-I", os.path.join(ROOT, "include"), "-I", build.CSRC,
                    os.path.join(ROOT, "tests", "cxx", "gemv_plan.cu"), "-o", exe, "-L", lib_dir, "-lkrk_cuda",
                    "-Xlinker", f"-rpath={lib_dir}"], check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
