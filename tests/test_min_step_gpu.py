"""The global time step's minimum (tests/cuda/min_step_check.cu): the FP32
comparison that picks a block's fastest faces never loses the smallest step,
also where a face's speed or length is outside FP32's range.

Bound: one product and the reciprocal, 2^-53 each, against a quotient and a
product: 2^-51 of the step.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
def test_block_minimum_against_fp64(gpu, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "min_step_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-I",
                    os.path.join(ROOT, "finitevolume_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cuda", "min_step_check.cu"), "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    rows = [line.split() for line in r.stdout.splitlines() if line]
    assert len(rows) == 10, r.stdout
    for f in rows:
        assert float(f[5]) <= 2.0 ** -51, f
