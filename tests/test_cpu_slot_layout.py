"""The layout of a mesh slot on the device (tests/layout_check.cpp)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = "/usr/local/cuda/include"


def test_slot_layout(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None or not os.path.isdir(CUDA):
        pytest.skip("no C++ compiler or CUDA headers")
    exe = str(tmp_path / "layout_check")
    cmd = [cxx, "-O1", "-std=c++17", "-I" + CUDA, "-I" + os.path.join(ROOT, "huji-rich_gb300", "csrc"),
           "-I" + os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "layout_check.cpp"), "-o", exe,
           "-L/usr/local/cuda/lib64", "-lcudart_static", "-ldl", "-lrt", "-lpthread"]
    subprocess.run(cmd, check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
