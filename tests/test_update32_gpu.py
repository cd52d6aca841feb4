"""The FP32-flux mode's Runge-Kutta stages against their operations in a fixed
order, bit for bit (tests/cuda/update32_check.cu): a last bit of the FP64 state
that the compiler's choice of multiply-adds moves becomes an FP32 rounding in
the cells' primitives, 2^-24 of them, and travels.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
def test_stages_keep_their_order_of_operations(gpu, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "update32_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-Xcompiler",
                    "-ffp-contract=off", "-I", os.path.join(ROOT, "finitevolume_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cuda", "update32_check.cu"), "-o", exe], check=True,
                   capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    rows = [line.split() for line in r.stdout.splitlines() if line]
    assert len(rows) == 6, r.stdout
    for f in rows:
        assert int(f[7]) == 0, f
