"""The fixed-point pieces of the second-order update (fixed.cuh: Runge-Kutta
stages of signed flux sums, sound speeds, local time steps, sums of squares) against long double, beside the FP64 forms
that they replace, on random operands; for the stages with the edges of the
formats among them: mantissas of all ones, cancelling sums, operands 2^30 apart.

Bounds.  Root mean square: no larger than the FP64 form's.  Largest: the one
rounding of the result, 2^-53 of it, and the integers' units, below 2^-56 of
the largest term (the states, the step factor times a flux); stages are at
most (3 + 1 + 4) / 4 and (1 + 2 + 8) / 3 times that, the others themselves.
Time steps: reciprocal, product and sum leave 2^-55.  Sums of 32 squares: each
within a unit of 2^-57 of the largest, 2^-52 together.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
def test_update_pieces_against_long_double(gpu, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "update_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-I",
                    os.path.join(ROOT, "finitevolume_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cuda", "update_check.cu"), "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    rows = [line.split() for line in r.stdout.splitlines() if line]
    if int(next(f[1] for f in rows if f[0] == "long_double_digits")) < 64:
        pytest.skip("long double is double on this host")
    eps = 2.0 ** -53
    size = {"stage1": 2.0, "stage2": 11.0 / 3.0, "sound": 1.0, "dt": 1.0, "squares": 1.0}
    units = {"dt": 1.0 / 4.0, "squares": 2.0}
    seen = 0
    for f in rows:
        if f[0] not in size:
            continue
        v = dict(zip(f[1::2], f[2::2]))
        assert int(v["taken"]) >= 0.99 * int(v["n"]), f
        assert float(v["rms_fixed"]) <= float(v["rms_fp64"]), f
        assert float(v["max_fixed"]) <= (size[f[0]] + units.get(f[0], 1.0 / 8.0)) * eps, f
        seen += 1
    assert seen == 5 * 3 + 2, r.stdout
