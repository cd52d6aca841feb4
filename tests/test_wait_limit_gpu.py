"""Which form of the first-order kernel runs, as split_launches() and persistent()
report it, and what a wait limit changes: the default build's launches of
phases give way to the cooperative kernels with their bounded waits, on a
local-dt mesh beyond the shared-memory dataflow form to the dataflow form with
the states in L2, and come back when the limit is back at its default.

Fields: the forms' arithmetic is the same, up to the compiler's contractions
(1e-13).
"""
import numpy as np
import pytest

from finitevolume_gb300 import capi, meshgen, solvers as S
from helpers import gpu_solver, rel_err, GAMMA

pytestmark = pytest.mark.gpu
DEFAULT = 2_000_000_000  # SM clock cycles


def _solver(size, local, **kw):
    M, aoa = 0.5, np.radians(2.0)
    r, u, v, p = 1.0, M * np.cos(aoa), M * np.sin(aoa), 1.0 / GAMMA
    bcs = [(0, [0.0] * 4), (3, list(S.from_primitive(r, u, v, p, GAMMA)))]
    return gpu_solver(meshgen.naca_ogrid(*size), bcs, {"mode": "free", "rho": r, "u": u, "v": v, "p": p}, "hllc",
                      cfl=0.5, local_dt=local, **kw)


@pytest.mark.parametrize("size,local,form,limited", [((64, 32), False, 1, 1), ((64, 32), True, 2, 2),
                                                     ((512, 330), True, 1, 2),
                                                     ((512, 400), True, 1, 2), ((512, 400), False, 1, 1)])
def test_forms_with_and_without_a_wait_limit(gpu, size, local, form, limited):
    """512 x 330: the blocks' own cells and faces fit in shared memory, with their neighbours' faces they do not."""
    a, b = _solver(size, local), _solver(size, local)
    assert a.persistent()[0] == form and a.split_launches() == (form == 1)
    b.set_wait_limit(DEFAULT + 1)
    assert b.persistent()[0] == limited and not b.split_launches() and b.persistent()[1] > 0
    for n in (1, 9, 35):
        ha, hb = a.run(n, history=True), b.run(n, history=True)
        assert rel_err(a.field(), b.field()) <= 1e-13
        np.testing.assert_allclose(ha, hb, rtol=1e-13, atol=0)
    # a wait that runs out ends the launch with an error; at the default limit the launches are back
    before = b.field()
    b.set_wait_limit(2_000_000, phantom_arrivals=1)
    with pytest.raises(capi.FVError) as e:
        b.run(1)
    assert e.value.status == capi.FV_ERR_TIMEOUT
    assert np.array_equal(b.field(), before)
    b.set_wait_limit(DEFAULT)
    assert b.persistent()[0] == form and b.split_launches() == (form == 1)
    a.set_field(before)
    b.set_field(before)
    assert np.array_equal(a.run(12, history=True), b.run(12, history=True))
    assert np.array_equal(a.field(), b.field())


def test_requested_forms(gpu):
    s = _solver((64, 32), False)
    s.set_persistent("barrier")
    assert s.persistent()[0] == 1 and not s.split_launches()
    s.set_persistent(False)
    assert s.persistent()[0] == 0 and not s.split_launches()
    s.set_persistent(True)
    assert s.persistent()[0] == 1 and s.split_launches()
    assert not _solver((64, 32), False, strict=True).split_launches()
    t = _solver((512, 400), True)
    t.set_persistent("barrier")
    t.set_wait_limit(DEFAULT + 1)
    assert t.persistent()[0] == 1 and not t.split_launches()
    t.run(2)


@pytest.mark.parametrize("size,local,split", [((64, 33), True, False), ((24, 9), True, False), ((64, 33), False, True), ((160, 75), False, True),
                                              ((160, 76), False, False), ((160, 76), True, False)])
def test_exact_flux_forms(gpu, size, local, split):
    """The exact Riemann flux: the dataflow form in L2 (24 x 9: its last block has no cells, and starts inside another's
    last warp), and one launch for the global step beyond 12,000 cells; against the grid-barrier form."""
    M, aoa = 0.5, np.radians(2.0)
    r, u, v, p = 1.0, M * np.cos(aoa), M * np.sin(aoa), 1.0 / GAMMA
    bcs = [(0, [0.0] * 4), (3, list(S.from_primitive(r, u, v, p, GAMMA)))]
    ic = {"mode": "free", "rho": r, "u": u, "v": v, "p": p}
    poly = meshgen.naca_ogrid(*size)
    a, b = (gpu_solver(poly, bcs, ic, "exact", cfl=0.5, local_dt=local) for _ in range(2))
    assert a.persistent()[0] == (2 if local else 1) and a.split_launches() == split
    b.set_persistent("barrier")
    assert b.persistent()[0] == 1 and not b.split_launches()
    for n in (1, 9):
        ha, hb = a.run(n, history=True), b.run(n, history=True)
        assert rel_err(a.field(), b.field()) <= 1e-13
        np.testing.assert_allclose(ha, hb, rtol=1e-13, atol=0)
