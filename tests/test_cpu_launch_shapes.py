"""The launch shapes' host rules (tests/shape_check.cpp): shapes that are set are
launched as given, built-in ones halved on small meshes."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = "/usr/local/cuda/include"


def test_launch_shapes(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None or not os.path.isdir(CUDA):
        pytest.skip("no C++ compiler or CUDA headers")
    exe = str(tmp_path / "shape_check")
    subprocess.run([cxx, "-O1", "-std=c++17", "-I" + CUDA, "-I" + os.path.join(ROOT, "huji-rich_gb300", "csrc"),
                    "-I" + os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "shape_check.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
