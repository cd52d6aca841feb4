"""The fixed-point gradient pass cell by cell (tests/cuda/grad_cells_check.cu):
that it serves every cell of at most 16 faces itself, instead of leaving it to
the FP64 pass (which would give the FP64 pass's errors, and so pass any bound
on them); its states beside boundaries, where lanes share ghosts by shuffles;
and the fallback to the cell's state where one is not positive.  Captured limiter
values: interior cells' errors relative to themselves (or 2^-7: what is below is
held to 2^-60) are no larger than the FP64 pass's, root mean square.

Bounds, in units of 2^-53 of the largest value times the weights'
amplification.  Interior cells: four roundings of a state, the root mean square
no larger than the FP64 pass's.  Beside boundaries a ghost adds its own error,
halved in the face's mean value: the characteristic farfield's density is a
fifth power, 5 times the roundings of its base (four) and 8 of the power itself,
its pressure two products more: (5 * 4 + 8 + 8) / 2 = 18, 24 with the state's.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
def test_cells_served_and_their_states(gpu, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "grad_cells_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-I",
                    os.path.join(ROOT, "finitevolume_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cuda", "grad_cells_check.cu"), "-o", exe], check=True,
                   capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    rows = [line.split() for line in r.stdout.splitlines() if line]
    if int(next(f[1] for f in rows if f[0] == "long_double_digits")) < 64:
        pytest.skip("long double is double on this host")
    eps = 2.0 ** -53
    seen = values = 0
    for f in rows:
        if f[0] == "long_double_digits":
            continue
        v = dict(zip(f[1::2], f[2::2]))
        if f[0].endswith("psi"):
            if int(v["boundary"]) == 0 and int(v["faces"]) <= 16:
                assert int(v["small"]) > 0, f
                assert float(v["rms_fixed"]) <= float(v["rms_fp64"]), f
            values += 1
            continue
        n, faces, boundary = int(v["n"]), int(v["faces"]), int(v["boundary"])
        assert int(v["served"]) == (n if faces <= 16 else 0), f
        assert int(v["declined"]) == n - int(v["served"]), f
        assert int(v["wrong"]) == 0, f
        # (a cell of nothing but boundary faces has no neighbour to overshoot towards)
        if f[0].endswith("open") and boundary < faces <= 16:
            assert int(v["fallback"]) > 0, f
        assert float(v["max_fixed"]) <= (4 if boundary == 0 else 24) * eps, f
        if boundary == 0:
            assert float(v["rms_fixed"]) <= float(v["rms_fp64"]), f
        seen += 1
    assert seen == 6 * 4 * 4 and values == 6 * 4 * 2, r.stdout
