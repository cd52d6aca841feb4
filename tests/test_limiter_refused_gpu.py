"""Limiter values of cells that the fixed-point gradient pass declines
(euler_o2_fixed.cuh: more than 16 faces; values out of range in one variable
only) against the FP64 pass's, which the same scheme with the exact Riemann
flux takes for every cell.

Tolerance: values jump by order one from cell to cell, so the limiter's
quotient sees the relative error of its two differences, each a few roundings of
the largest value: 1e-10 leaves 2^19 roundings of 2^-53 for differences down to
2^-19 of the values.
"""
import numpy as np
import pytest

from finitevolume_gb300 import meshgen, solvers as S
from finitevolume_gb300.fvmesh import PolyMesh
from helpers import GAMMA

pytestmark = pytest.mark.gpu


def mesh_with_big_cell(n=20, at=(6, 7), size=6):
    """n x n quads, a block of size x size of them merged into one cell of 4 size faces."""
    p = meshgen.cartesian(n, n)
    quads = p.cell_nodes.reshape(-1, 4)
    i0, j0 = at
    inside = np.zeros((n, n), bool)
    inside[j0:j0 + size, i0:i0 + size] = True
    node = lambda i, j: j * (n + 1) + i  # noqa: E731
    ring = [node(i, j0) for i in range(i0, i0 + size)] + [node(i0 + size, j) for j in range(j0, j0 + size)]
    ring += [node(i, j0 + size) for i in range(i0 + size, i0, -1)] + [node(i0, j) for j in range(j0 + size, j0, -1)]
    cells = [list(q) for q in quads[~inside.ravel()]] + [ring]
    used = np.unique(np.concatenate([np.asarray(c) for c in cells]))
    new = np.full(p.n_nodes, -1)
    new[used] = np.arange(used.size)
    off = np.concatenate([[0], np.cumsum([len(c) for c in cells])])
    return PolyMesh(p.nodes[used], off.astype(np.int64), new[np.concatenate([np.asarray(c) for c in cells])].astype(np.int32),
                    new[p.bedges].astype(np.int32), p.bpatch, p.patch_names)


def solver(poly, flux, limiter, **kw):
    T = S.EulerBoundaryType
    far = S.from_primitive(1.0, 0.3, 0.2, 1.0 / GAMMA, GAMMA)
    bcs = [S.EulerBoundaryCondition(T.Wall), S.EulerBoundaryCondition(T.CharacteristicFarfield, far),
           S.EulerBoundaryCondition(T.Outflow), S.EulerBoundaryCondition(T.Farfield, far)]
    ic = S.EulerInitialCondition(S.EulerICMode.Freestream, rho=1.0, u=0.3, v=0.2, p=1.0 / GAMMA)
    return S.EulerFVMSolver(S.Mesh(poly), bcs, GAMMA, 0.2, ic, flux, order=2, rk_stages=3, local_dt=True,
                            gradient=S.GradientScheme.LeastSquares, limiter=limiter, **kw)


def jumps(poly, seed, tiny_v=False):
    rng = np.random.default_rng(seed)
    n = poly.n_cells
    r, u, p = 1.0 + rng.random(n), rng.random(n) - 0.5, 0.5 + rng.random(n)
    v = (rng.random(n) - 0.5) * (1e-300 if tiny_v else 1.0)
    return np.stack([r, r * u, r * v, p / (GAMMA - 1.0) + 0.5 * r * (u * u + v * v)], -1)


@pytest.mark.parametrize("limiter", [S.Limiter.BarthJespersen, S.Limiter.Venkatakrishnan])
@pytest.mark.parametrize("big", [True, False])
@pytest.mark.parametrize("tiny_v", [False, True])
def test_captured_values_of_declined_cells(gpu, limiter, big, tiny_v):
    poly = mesh_with_big_cell() if big else meshgen.cartesian(20, 20)
    U = jumps(poly, 3, tiny_v)
    psi = []
    for flux in (S.NumericalFluxScheme.HLLC, S.NumericalFluxScheme.Exact):
        s = solver(poly, flux, limiter)
        s.set_field(U)
        s.freeze_limiter()
        psi.append(s.limiter_values())
    if tiny_v:  # every cell is declined for its v alone, whose own value is rounding noise
        psi = [np.delete(p, 2, axis=1) for p in psi]
    assert (psi[1] < 0.9).mean() > 0.2
    np.testing.assert_allclose(psi[0], psi[1], rtol=0, atol=1e-10)


@pytest.mark.parametrize("k", [-1.0, -0.0, 0.0])
def test_negative_and_zero_venkat_k(gpu, k):
    """A negative K makes eps^2 = (K h)^3 negative, which only the FP64 pass forms.  With eps^2 about -1e-4 the
    quotient's denominator comes near zero at a few cells: 1e-8 leaves it 2^-26 of the squared differences."""
    poly = meshgen.cartesian(20, 20)
    U = jumps(poly, 5)
    psi = []
    for flux in (S.NumericalFluxScheme.HLLC, S.NumericalFluxScheme.Exact):
        s = solver(poly, flux, S.Limiter.Venkatakrishnan, venkat_k=k)
        s.set_field(U)
        s.freeze_limiter()
        psi.append(s.limiter_values())
    np.testing.assert_allclose(psi[0], psi[1], rtol=1e-8, atol=1e-8)
