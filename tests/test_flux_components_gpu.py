"""The fixed-point fluxes component by component (tests/cuda/
flux_components_check.cu).  Block fixed point holds every component to a place
of the face's scale: a component far below that scale (a normal near an axis
beside a small velocity) keeps fewer bits of its own than FP64's, which is
printed but not bounded.

Bound: each component's root mean square error, of the face's scale, is that of
two roundings (the conversion and the product with the length) of at most 6
times the scale, (1 / (gamma - 1) + 1 / 2) (1 + Mach): 6 sqrt(2 / 3) < 5 roundings
of 2^-53.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
def test_components_of_the_fluxes(gpu, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "flux_components_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-I",
                    os.path.join(ROOT, "finitevolume_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cuda", "flux_components_check.cu"), "-o", exe], check=True,
                   capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    print(r.stdout)
    rows = [line.split() for line in r.stdout.splitlines() if line]
    if int(next(f[1] for f in rows if f[0] == "long_double_digits")) < 64:
        pytest.skip("long double is double on this host")
    rows = [f for f in rows if f[0] in ("rusanov", "hllc")]
    assert len(rows) == 2 * 3 * 4, r.stdout
    for f in rows:
        v = dict(zip(f[2::2], f[3::2]))
        assert int(v["taken"]) == int(v["n"]), f
        assert float(v["scale_fixed"]) <= 5 * 2.0 ** -53, f
