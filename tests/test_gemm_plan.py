"""The tile and split plan of the prefill GEMM, on the host: devices that hold few clusters of a size, or none."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_every_tile_is_planned_whatever_the_device_holds(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = str(tmp_path / "gemm_plan")
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "kraken_b200", "csrc"), os.path.join(ROOT, "tests", "cxx", "gemm_plan.cpp"),
                    "-o", exe], check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
