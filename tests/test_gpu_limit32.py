"""The FP32 limiter over the range of a cell's reconstructed values
(huji-rich_gb300/csrc/rg_limit32.cuh) against the limiter face by face, bit for
bit, and the monotone FP32 quotient it rests on (tests/limit32_check.cu)."""
import json
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
def test_range_limiter_bitwise_equal(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "limit32_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "-I" + os.path.join(ROOT, "huji-rich_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "limit32_check.cu"), "-o", exe], check=True)
    for seed in (1, 2):
        r = subprocess.run([exe, str(seed)], capture_output=True, text=True, timeout=300)
        res = json.loads(r.stdout.strip().splitlines()[-1])
        assert res["not_monotone"] == 0 and res["mismatches"] == 0 and r.returncode == 0, res
        assert res["limited"] > 0.05 * res["cases"], res
