"""Device memory of a second-order FP64 solver: the fixed-point geometry (132
bytes a quad) takes the place of arrays that the FP64 passes needed (the limited
gradients, 64 bytes a cell, and the limiter values), so that a mesh that filled
the card still fits.

Bound: 904 bytes a cell were needed before, 36 more are; 960 leaves room for the
allocations' granularity and the mesh's boundary.
"""
import pytest

from finitevolume_gb300 import meshgen, solvers as S
from helpers import GAMMA

pytestmark = pytest.mark.gpu


def test_bytes_a_cell(gpu):
    torch = pytest.importorskip("torch")
    poly = meshgen.cartesian(1024, 1000)
    mesh = S.Mesh(poly)
    bcs = [S.EulerBoundaryCondition(S.EulerBoundaryType.Outflow)] * 4
    ic = S.EulerInitialCondition(S.EulerICMode.Freestream, rho=1.0, u=0.4, v=0.3, p=1.0 / GAMMA)
    torch.zeros(1, device="cuda")
    free = torch.cuda.mem_get_info()[0]
    s = S.EulerFVMSolver(mesh, bcs, GAMMA, 0.3, ic, S.NumericalFluxScheme.HLLC, order=2, rk_stages=3, local_dt=True)
    used = (free - torch.cuda.mem_get_info()[0]) / poly.n_cells
    s.run(2)
    assert used <= 960, used
