"""The first-order barrier form's phases as launches of their own (the default
build's global-dt path, and its local-dt one on meshes beyond the dataflow
form) against the barrier kernel that set_persistent("barrier") asks for: the
same arithmetic per face, cell and norm tile, so fields and histories agree to
rounding (1e-13: the compiler may contract differently in the two).

Sizes: one block of cells with a partial tile, several, and a local-dt mesh
beyond the dataflow form.  Step counts: around the eight steps whose norm
partials are kept and beyond a graph of 32.  A wait limit that is set brings
the barrier kernel (and its FV_ERR_TIMEOUT) back.
"""
import numpy as np
import pytest

from finitevolume_gb300 import capi, meshgen, solvers as S
from helpers import gpu_solver, rel_err, GAMMA

pytestmark = pytest.mark.gpu


def _case(local):
    M, aoa = 0.5, np.radians(2.0)
    r, u, v, p = 1.0, M * np.cos(aoa), M * np.sin(aoa), 1.0 / GAMMA
    st = list(S.from_primitive(r, u, v, p, GAMMA))
    return [(0, [0.0] * 4), (3 if local else 1, st)], {"mode": "free", "rho": r, "u": u, "v": v, "p": p}


@pytest.mark.parametrize("flux", ["rusanov", "hllc", "exact"])
@pytest.mark.parametrize("size,local,steps", [((16, 8), False, (1, 7, 9)), ((64, 33), False, (8, 1, 40)),
                                              ((512, 400), True, (9, 35))])
def test_split_matches_barrier_form(gpu, flux, size, local, steps):
    poly = meshgen.naca_ogrid(*size)
    bcs, ic = _case(local)
    a = gpu_solver(poly, bcs, ic, flux, cfl=0.5, local_dt=local)
    b = gpu_solver(poly, bcs, ic, flux, cfl=0.5, local_dt=local)
    b.set_persistent("barrier")
    assert a.persistent()[0] == 1 and b.persistent()[0] == 1
    for n in steps:
        ha, hb = a.run(n, history=True), b.run(n, history=True)
        assert rel_err(a.field(), b.field()) <= 1e-13
        np.testing.assert_allclose(ha, hb, rtol=1e-13, atol=0)


def test_wait_limit_brings_the_barrier_kernel_back(gpu):
    poly = meshgen.naca_ogrid(64, 32)
    bcs, ic = _case(False)
    a = gpu_solver(poly, bcs, ic, "hllc", cfl=0.5)
    a.run(3)
    before = a.field()
    a.set_wait_limit(2_000_000, phantom_arrivals=1)
    with pytest.raises(capi.FVError) as e:
        a.run(3)
    assert e.value.status == capi.FV_ERR_TIMEOUT
    assert np.array_equal(a.field(), before)
    a.set_wait_limit(2_000_000_000, phantom_arrivals=0)
    b = gpu_solver(poly, bcs, ic, "hllc", cfl=0.5)
    b.run(3)
    assert np.array_equal(a.run(3, history=True), b.run(3, history=True))
    assert np.array_equal(a.field(), b.field())
