"""Moving-mesh contexts whose pressure has no multigrid hierarchy: meshes too
small to coarsen, and a pressure without a Dirichlet boundary. They are set up
and solved by the Jacobi CG.
"""
import numpy as np
import pytest

from pfem2_b200 import _abi as A
from pfem2_b200 import cases
from tests.helpers import rel_l2
from tests.test_gpu_parity import make_pair, set_vel, smooth_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny", [(2, 2), (4, 2), (6, 3), (32, 12)])
def test_small_moving_mesh(nx, ny, prec):
    """one FEM step against the oracle; the largest mesh has a hierarchy"""
    sp = cases.poiseuille_2d(nx=nx, ny=ny)
    sp.case.dt = 0.05
    sp.case.vel_tol = 1e-13
    sp.case.p_tol = 1e-12
    g, o = make_pair(sp, prec, moving_mesh=True)
    set_vel(g, o, sp, smooth_field(sp.mesh.vertices, 0.5))
    g.fem_step()
    o.fem_step(1)
    g.stats()  # raises unless every solve converged
    assert (g.solver_sizes()["n1"] > 0) == (nx == 32)
    for f in (A.FIELD_PRED_VX, A.FIELD_PRED_VY, A.FIELD_P, A.FIELD_VX, A.FIELD_VY):
        assert rel_l2(g.field(f), o.field(f)) <= 1e-8, f


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("nx,ny", [(6, 3), (64, 16)])
def test_moving_mesh_without_dirichlet_pressure(nx, ny, prec):
    """the pressure matrix is singular, and with an inflow its right-hand side
    need not be in its range: the solve ends at max_iter and says so"""
    sp = cases.poiseuille_2d(nx=nx, ny=ny)
    sp.case.n_dirichlet[3] = 0
    sp.case.max_iter = 500
    sp.case.vel_rtol = sp.case.p_rtol = 1e-9
    sp.case.vel_tol = sp.case.p_tol = 0.0
    g, _ = make_pair(sp, prec, moving_mesh=True)
    assert g.solver_sizes()["n1"] == 0
    for d, v in enumerate(smooth_field(sp.mesh.vertices, 0.5)):
        g.set_field(A.FIELD_VX + d, v)
    try:
        g.fem_step()
    except Exception as e:
        assert e.status == A.NOT_CONVERGED
    assert g.stats(check=False)["status"] in (A.OK, A.NOT_CONVERGED)
    for f in (A.FIELD_P, A.FIELD_VX, A.FIELD_VY):
        assert np.isfinite(g.field(f)).all()
