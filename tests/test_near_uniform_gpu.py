"""Uniform flows and flows just beside them through the viscous solver's default
build, whose Rusanov mass flux takes another form where both densities are
equal (viscous_fast.cuh): residual histories against the strict build's.

Bound: a cell's residual sums four fluxes of order one times a length of 1/64, a
few roundings of 2^-53 each; over 6,144 cells the norms differ by less than
sqrt(6144) * 32 * 2^-53 / 64 < 1e-14, in the energy as in the others, and the
differences decay with the perturbation.
"""
import numpy as np
import pytest

from finitevolume_gb300 import meshgen, solvers as S
from helpers import GAMMA

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flux", [S.NumericalFluxScheme.Rusanov, S.NumericalFluxScheme.HLLC])
@pytest.mark.parametrize("size", [0.0, 2.0 ** -52, 1e-14, 1e-9])
def test_residuals_beside_equal_densities(gpu, flux, size):
    r, u, v, p = 1.0, 0.5, 0.1, 1.0 / GAMMA
    poly = meshgen.cartesian(96, 64, 1.5, 1.0)
    far = S.NSBoundaryCondition(S.NSBoundaryType.Farfield, farfield_state=list(S.from_primitive(r, u, v, p, GAMMA)))
    ic = S.EulerInitialCondition(S.EulerICMode.Freestream, rho=r, u=u, v=v, p=p)
    q = r + size * np.random.default_rng(0).standard_normal(poly.n_cells)
    U = np.stack([q, q * u, q * v, p / (GAMMA - 1.0) + 0.5 * q * (u * u + v * v)], -1)
    h = []
    for strict in (True, False):
        s = S.NavierStokesFVMSolver(S.Mesh(poly), [far] * 4, GAMMA, 287.0, 1e-3, 0.72, 0.5, ic, flux,
                                    S.GradientScheme.GreenGauss, strict=strict)
        s.set_field(U)
        h.append(s.run(20, history=True))
    assert np.abs(h[1] - h[0]).max() <= 1e-14
