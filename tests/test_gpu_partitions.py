"""The persistent solvers' partitions against the FP64 oracle: one cluster or a
grid of blocks, one or several warps to a row slice, one or two blocks per SM,
few long and many short slice runs, the pressure hierarchy with narrow and wide
restriction rows and with and without a published level 1 (3D). Bars as for the
parity of one FEM step: both sides solve to absolute residuals of 1e-13
(velocity) and 1e-12 (pressure), which separates the fields by less than 1e-8.
"""
import numpy as np
import pytest

from pfem2_b200 import _abi as A
from pfem2_b200 import cases
from tests.helpers import rel_l2
from tests.test_gpu_parity import make_pair, set_vel, smooth_field

pytestmark = pytest.mark.gpu

CG, BICG = A.SOLVER_CG, A.SOLVER_BICGSTAB


@pytest.mark.parametrize("size,prec,kind,tuning,wide", [
    ((32, 12), "mixed", CG, {}, 0),                                               # one cluster
    ((32, 12), "fp64", BICG, {"vel_tile_slices": 40}, 0),                         # one block, items in two rounds
    ((128, 48), "fp64", CG, {}, 0),                                               # grid, split rows
    ((128, 48), "fp64", BICG, {"vel_tile_slices": 1, "vel_blocks_per_sm": 1}, 1),  # one slice a block
    ((128, 48), "mixed", BICG, {"vel_tile_slices": 2, "vel_blocks_per_sm": 2, "p_blocks_per_sm": 2}, 0),
    ((40, 10, 10), "fp64", BICG, {}, 0),                                          # three components, split rows
    ((40, 10, 10), "mixed", CG, {"vel_tile_slices": 3}, 1),
    ((40, 10, 10), "fp64", CG, {"vel_blocks_per_sm": 2, "p_blocks_per_sm": 2}, 0),
])
def test_fem_step_partitions(monkeypatch, size, prec, kind, tuning, wide):
    if wide:
        monkeypatch.setenv("PFEM2_MG_WIDE_MIN", "1")
    if len(size) == 2:
        sp = cases.poiseuille_2d(nx=size[0], ny=size[1])
        # (at a tenth of this step the FP64 rounding of b - A x on the 6k rows,
        # about 2e-12, lies above the pressure tolerance)
        sp.case.dt = 0.05
    else:
        sp = cases.pipe_3d(nx=size[0], ny=size[1], nz=size[2])
        sp.case.dt = 0.002
    dim = len(size)
    sp.case.vel_tol = 1e-13
    sp.case.p_tol = 1e-12
    sp.case.vel_solver = kind
    g, o = make_pair(sp, prec, tuning=tuning)
    set_vel(g, o, sp, smooth_field(sp.mesh.vertices, 0.5))
    g.fem_step()
    o.fem_step(1)
    it = np.array(g.stats()["iters"])
    assert it[0] > 0 and it[3] > 0
    for fld in [A.FIELD_PRED_VX + d for d in range(dim)] + [A.FIELD_P] + [A.FIELD_VX + d for d in range(dim)]:
        e = rel_l2(g.field(fld), o.field(fld))
        assert e <= 1e-8, (fld, e)


def test_bicgstab_of_rounding_sized_components():
    """a pipe whose cross components are rounding noise, every solve to 1e-11
    of its right-hand side: no BiCGStab solve loses its direction and runs on
    towards max_iter (the solves that do not take 30 to 90 iterations)"""
    sp = cases.pipe_3d(nx=48, ny=12, nz=12)
    sp.case.vel_solver = BICG
    sp.case.vel_tol = sp.case.p_tol = 0.0
    sp.case.vel_rtol = sp.case.p_rtol = 1e-11
    g, _ = make_pair(sp, "fp64")
    g.seed_particles(sp.q, seed=sp.seed, jitter=sp.jitter)
    for _ in range(8):
        g.step()
        st = g.stats()
        it = st["iters"]
        assert st["status"] == A.OK and max(it[:3] + it[4:7]) <= 500
