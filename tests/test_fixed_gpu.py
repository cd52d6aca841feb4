"""The fixed-point gradient, limiter and flux passes of the second-order path
(finitevolume_gb300/csrc/fixed.cuh, euler_o2_fixed.cuh) against long double,
beside the FP64 forms that they replace: on random face states (smooth,
jumps, low Mach numbers, velocities and normals along the axes, four gammas,
scales from 2^-30 to 2^30; the same as the first-order kernel's conserved
states) and random cells of 3 to 16 faces (and 18, which
the FP64 form takes).

Bounds.  Root mean square: no larger than the FP64 form's.  Largest: a flux
is at most eight roundings of 2^-53 of the face's own scale (r q^3 for the
energy, q the larger of speed and sound speed), whose factors here reach
1/(gamma - 1) + 1/2 <= 5.5 times (1 + Mach) <= 4 times it; a face state at
most four roundings of the largest value it is formed from.  States outside
the ranges are refused, every one.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
def test_fixed_point_passes_against_long_double(gpu, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "fixed_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-I",
                    os.path.join(ROOT, "finitevolume_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cuda", "fixed_check.cu"), "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    rows = [line.split() for line in r.stdout.splitlines() if line]
    digits = int(next(f[1] for f in rows if f[0] == "long_double_digits"))
    if digits < 64:
        pytest.skip("long double is double on this host")
    eps = 2.0 ** -53
    seen = 0
    for f in rows:
        if f[0] == "long_double_digits":
            continue
        v = dict(zip(f[1::2], f[2::2]))
        if "refused" in v:
            assert int(v["accepted"]) == 0, f
            continue
        flux = not f[0].startswith("grad")
        # taken: all but jumps beyond the ratios; all cells but those of 18 faces
        assert int(v["taken"]) >= (0.97 if flux else 0.87) * int(v["n"]), f
        assert float(v["rms_fixed"]) <= float(v["rms_fp64"]), f
        assert float(v["max_fixed"]) <= (8 * 5.5 * 4 if flux else 4) * eps, f
        seen += 1
    assert seen == 2 * 4 * 2 * 4 + 8, r.stdout
