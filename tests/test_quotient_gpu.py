"""fvconv::quotient, the division of the diffusion solver's face pass by a
prepared reciprocal: the IEEE quotient bit for bit."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
def test_quotient_is_the_ieee_division(gpu, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "quotient_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-I",
                    os.path.join(ROOT, "finitevolume_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cuda", "quotient_check.cu"), "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.split() == ["checked", str(2 ** 28), "mismatch", "0"], r.stdout
