"""Batches of instances of one to three row slices (32 rows each), of which a
block of the velocity solves' grid owns parts of many: they set up, whatever
least number of slices per block is asked for, and every instance gets the
solution of a context of its own.
"""
import numpy as np
import pytest

from pfem2_b200 import _abi as A
from pfem2_b200 import cases
from pfem2_b200.solver import Solver
from tests.helpers import rel_l2
from tests.test_gpu_parity import smooth_field

pytestmark = pytest.mark.gpu


def spec(dim, size):
    if dim == 2:
        sp = cases.poiseuille_2d(nx=size[0], ny=size[1])
    else:
        sp = cases.pipe_3d(nx=size[0], ny=size[1], nz=size[2])
        sp.case.p_solver = A.SOLVER_BICGSTAB  # (too small for a multigrid hierarchy)
        sp.case.dt = 0.002
    sp.case.vel_tol = 1e-13
    sp.case.p_tol = 1e-12
    return sp


def step(specs, tuning):
    s = Solver(specs, precision=A.PREC_FP64, tuning=tuning)
    for i, sp in enumerate(specs):
        for d, v in enumerate(smooth_field(sp.mesh.vertices, 0.5)):
            s.set_field(A.FIELD_VX + d, v, i)
    s.fem_step()
    s.stats()
    out = [[s.field(A.FIELD_VX + d, i) for d in range(sp.mesh.dim)] + [s.field(A.FIELD_P, i)]
           for i, sp in enumerate(specs)]
    s.close()
    return out


@pytest.mark.parametrize("dim,sizes,n,tuning", [
    (2, [(15, 3)], 2340, None),                       # 2 slices each: up to 9 instances of 2 systems in a block
    (2, [(15, 3)], 100, {"vel_tile_slices": 16}),     # 16 slices touch 9 instances
    (2, [(15, 3)], 100, {"vel_tile_slices": 4096}),   # one block could not hold the batch
    (2, [(15, 3), (23, 3), (40, 20)], 30, {"vel_tile_slices": 64, "vel_blocks_per_sm": 1}),  # uneven
    (3, [(5, 2, 2)], 1560, None),                     # 2 slices: up to 7 instances of 3 systems
    (3, [(2, 2, 2), (5, 2, 2), (7, 3, 2)], 60, {"vel_tile_slices": 40}),
])
def test_batch_of_small_instances(dim, sizes, n, tuning):
    kinds = [spec(dim, z) for z in sizes]
    alone = [step([sp], None)[0] for sp in kinds]
    got = step([kinds[i % len(kinds)] for i in range(n)], tuning)
    for i, fields in enumerate(got):
        for f, g in zip(alone[i % len(kinds)], fields):
            assert rel_l2(g, f) <= 1e-8, i
