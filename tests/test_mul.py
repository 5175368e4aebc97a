"""The correctly rounded FP64 product of huji-rich_gb300/csrc/rg_mul.cuh
(integer pipes), host and device builds, against the IEEE product, bit for
bit (tests/mul_check.cu, operand families in tests/mul_cases.h)."""
import json
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "mul_check.cu")
INC = ["-I" + os.path.join(ROOT, "huji-rich_gb300", "csrc"), "-I" + os.path.join(ROOT, "tests")]


def check(exe, n, seed):
    r = subprocess.run([exe, str(n), str(seed)], capture_output=True, text=True, timeout=900)
    res = json.loads(r.stdout.strip().splitlines()[-1])
    assert res["mismatches"] == 0 and r.returncode == 0, res
    # of the six families one is all bit patterns (an eighth of them not
    # normal products), one spans every exponent, one sits at the range's ends
    assert res["cases"] > 5 * n and res["fast"] > 0.6 * res["cases"], res


@pytest.mark.parametrize("seed", [1, 2])
def test_host_product_bitwise_equal_to_ieee(tmp_path, seed):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "mul_check")
    subprocess.run([cxx, "-x", "c++", "-O2", "-std=c++17", "-ffp-contract=off"] + INC + [SRC, "-o", exe], check=True)
    check(exe, 500000, seed)


@pytest.mark.gpu
def test_device_product_bitwise_equal_to_ieee(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "mul_check_gpu")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17"] + INC + [SRC, "-o", exe],
                   check=True)
    check(exe, 1000000, 3)
