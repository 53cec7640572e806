"""Jacobi solves whose blocks keep the items' partial sums in global memory, as
very large systems do: PFEM2_PARTIALS_MAX=0 takes that form at any size where
no warps share an item. Bars as for the parity of one FEM step.
"""
import pytest

from pfem2_b200 import _abi as A
from pfem2_b200 import cases
from tests.helpers import rel_l2
from tests.test_gpu_parity import make_pair, set_vel, smooth_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,prec,kind,tuning", [
    ((32, 12), "fp64", A.SOLVER_BICGSTAB, {"vel_tile_slices": 40}),  # one block, 28 items for 24 warps
    ((97, 40), "mixed", A.SOLVER_CG, {"vel_tile_slices": 8}),
    ((97, 40), "fp64", A.SOLVER_CG, {"vel_tile_slices": 13, "vel_blocks_per_sm": 1}),
    ((24, 10, 10), "mixed", A.SOLVER_BICGSTAB, {"vel_tile_slices": 9}),
])
@pytest.mark.parametrize("limit", [None, 0])
def test_fem_step(monkeypatch, limit, size, prec, kind, tuning):
    if limit is not None:
        monkeypatch.setenv("PFEM2_PARTIALS_MAX", str(limit))
    if len(size) == 2:
        sp = cases.poiseuille_2d(nx=size[0], ny=size[1])
        sp.case.dt = 0.05
    else:
        sp = cases.pipe_3d(nx=size[0], ny=size[1], nz=size[2])
        sp.case.dt = 0.002
    sp.case.vel_tol = 1e-13
    sp.case.p_tol = 1e-12
    sp.case.vel_solver = sp.case.p_solver = kind
    g, o = make_pair(sp, prec, tuning=tuning)
    set_vel(g, o, sp, smooth_field(sp.mesh.vertices, 0.5))
    g.fem_step()
    o.fem_step(1)
    dim = sp.mesh.dim
    for f in [A.FIELD_PRED_VX + d for d in range(dim)] + [A.FIELD_P] + [A.FIELD_VX + d for d in range(dim)]:
        assert rel_l2(g.field(f), o.field(f)) <= 1e-8, f
