"""The sixth root of the turbulence model's destruction term (rans.cu, default
build: inv_root6) against long double over its whole range of exponents, and
beyond it, where the library's roots take over.

Bound: the last multiply-add's rounding and 5/6 of one from y^6's five make less
than 2^-52; the library's two roots and a division at most 2^-51.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
def test_sixth_root_over_its_range(gpu, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "root6_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "--expt-relaxed-constexpr",
                    "-I", os.path.join(ROOT, "finitevolume_gb300", "csrc"), "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "cuda", "root6_check.cu"), "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    rows = [line.split() for line in r.stdout.splitlines() if line]
    if int(next(f[1] for f in rows if f[0] == "long_double_digits")) < 64:
        pytest.skip("long double is double on this host")
    rows = [f for f in rows if f[0] == "exponent"]
    assert len(rows) == 176, r.stdout
    for f in rows:
        assert float(f[3]) <= 2.0 ** (-52 if -60 <= int(f[1]) <= 100 else -51), f
