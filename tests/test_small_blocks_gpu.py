"""Edges of three work splits.

- The shared-memory dataflow form on meshes of one to four blocks: one block
  without a mailbox (32 cells), blocks with a ragged last warp (36, 72), against
  the barrier form: bit for bit in strict mode, to 1e-13 in the default build
  (whose compiler may contract differently in the two kernels).
- The batched norms' chunks of 1,024 cells: instances of a multiple of it, a few
  below, a few above, and one small, against the standalone solver's norms
  (1e-12: sums of at most 2,048 squares, 2048 * 2^-53 on either side).
- The gradient pass's order of tiles on a mesh with polygons, whose last tile is
  ragged, under launch shapes that are and are not multiples of a tile's 128
  lanes: every cell is served, so fields are the same bits.
"""
import numpy as np
import pytest

from finitevolume_gb300 import meshgen, solvers as S
from helpers import gpu_solver, rel_err, GAMMA

pytestmark = pytest.mark.gpu


def _fs(M, aoa):
    a = np.radians(aoa)
    return 1.0, M * np.cos(a), M * np.sin(a), 1.0 / GAMMA


@pytest.mark.parametrize("strict", [True, False])
@pytest.mark.parametrize("flux", ["rusanov", "hllc"])
@pytest.mark.parametrize("size", [(8, 4), (12, 3), (12, 6), (16, 8)])
def test_shared_memory_form_on_few_blocks(gpu, size, flux, strict):
    poly = meshgen.naca_ogrid(*size)
    r, u, v, p = _fs(0.3, 2.0)
    bcs = [(0, [0.0] * 4), (3, list(S.from_primitive(r, u, v, p, GAMMA)))]
    ic = {"mode": "free", "rho": r, "u": u, "v": v, "p": p}
    a = gpu_solver(poly, bcs, ic, flux, cfl=0.4, local_dt=True, strict=strict)
    b = gpu_solver(poly, bcs, ic, flux, cfl=0.4, local_dt=True, strict=strict)
    b.set_persistent("barrier")
    assert a.persistent()[0] == 2 and b.persistent()[0] == 1
    for n in (1, 2, 33):
        ha, hb = a.run(n, history=True), b.run(n, history=True)
        if strict:
            assert np.array_equal(a.field(), b.field()) and np.array_equal(ha, hb)
        else:
            assert rel_err(a.field(), b.field()) <= 1e-13
            np.testing.assert_allclose(ha, hb, rtol=1e-13, atol=0)


def test_tile_order_serves_every_cell_at_any_launch_shape(gpu):
    poly = meshgen.naca_mixed(32, 16, seed=0)
    assert poly.n_cells % 32 != 0
    fs = _fs(0.5, 1.0)
    bcs = [S.EulerBoundaryCondition(S.EulerBoundaryType.Wall),
           S.EulerBoundaryCondition(S.EulerBoundaryType.CharacteristicFarfield, S.from_primitive(*fs, GAMMA))]
    ic = S.EulerInitialCondition(S.EulerICMode.Freestream, rho=fs[0], u=fs[1], v=fs[2], p=fs[3])
    fields = []
    for shape in (128, 160, 224, 480, 512):
        s = S.EulerFVMSolver(S.Mesh(poly), bcs, GAMMA, 1.0, ic, S.NumericalFluxScheme.HLLC, order=2, rk_stages=3,
                             local_dt=True)
        s.set_launch(shape, 128, 128)
        s.run(5)
        fields.append(s.field())
    assert all(np.array_equal(f, fields[0]) for f in fields[1:])


def test_batched_norms_at_the_chunk_edges(gpu):
    sizes = [(16, 8), (32, 32), (34, 30), (38, 27), (64, 32)]
    meshes = [S.Mesh(meshgen.naca_ogrid(*s)) for s in sizes]
    fss = [_fs(0.3 + 0.05 * i, 1.0) for i in range(len(sizes))]
    b = S.BatchSolver(meshes, [S.EulerBoundaryType.Wall, S.EulerBoundaryType.CharacteristicFarfield], fss)
    b.run(3)
    norms = b.status()[2]
    for i, (m, fs) in enumerate(zip(meshes, fss)):
        bcs = [S.EulerBoundaryCondition(S.EulerBoundaryType.Wall),
               S.EulerBoundaryCondition(S.EulerBoundaryType.CharacteristicFarfield, S.from_primitive(*fs, GAMMA))]
        ic = S.EulerInitialCondition(S.EulerICMode.Freestream, rho=fs[0], u=fs[1], v=fs[2], p=fs[3])
        s = S.EulerFVMSolver(m, bcs, GAMMA, 1.2, ic, S.NumericalFluxScheme.HLLC, order=2, rk_stages=3, local_dt=True)
        s.run(3)
        np.testing.assert_allclose(norms[i], s.residual().as_array(), rtol=1e-12)
