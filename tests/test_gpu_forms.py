"""Which form of the solvers each size takes. tests/test_gpu_partitions.py
compares the fields of these sizes with the oracle; here the intended forms are
named, so that a changed rule that drops one of them is seen.
"""
import pytest

from pfem2_b200 import _abi as A
from pfem2_b200 import cases
from pfem2_b200.solver import Solver
from tests.helpers import solver_kw

pytestmark = pytest.mark.gpu

CG, BICG = A.SOLVER_CG, A.SOLVER_BICGSTAB


def forms(specs, prec, kind, tuning=None):
    for sp in specs:
        sp.case.vel_solver = kind
    s = Solver(specs, tuning=tuning, **solver_kw(prec))
    out = s.solver_forms()
    s.close()
    return out


def spec(size):
    if len(size) == 2:
        return cases.poiseuille_2d(nx=size[0], ny=size[1])
    return cases.pipe_3d(nx=size[0], ny=size[1], nz=size[2])


def subset(want, got):
    return {k: got[k] for k in want} == want


@pytest.mark.parametrize("size,prec,kind,tuning,wide,vel,p", [
    ((32, 12), "mixed", CG, {}, 0, dict(cluster=1, warps_per_slice=1), dict(blocks_per_sm=1, staged=0)),
    ((32, 12), "fp64", BICG, {"vel_tile_slices": 40}, 0, dict(cluster=0, blocks=1, warps_per_slice=1), {}),
    ((128, 48), "fp64", CG, {}, 0, dict(cluster=0, blocks_per_sm=2, warps_per_slice=2), {}),
    ((128, 48), "fp64", BICG, {"vel_tile_slices": 1, "vel_blocks_per_sm": 1}, 1,
     dict(cluster=0, blocks_per_sm=1), dict(blocks_per_sm=2)),
    ((128, 48), "mixed", BICG, {"vel_tile_slices": 2, "vel_blocks_per_sm": 2, "p_blocks_per_sm": 2}, 0,
     dict(blocks_per_sm=2), dict(blocks_per_sm=2)),
    # rows of 27 entries: 6 items to 24 warps, 9 entries a warp (2 rounds of 5 loads)
    ((40, 10, 10), "fp64", BICG, {}, 0, dict(cluster=0, warps_per_slice=3),
     dict(blocks_per_sm=1, level1_published=1, restriction_lanes=32)),
    # 9 items, 14 entries a warp (2 rounds of 9 loads instead of 3)
    ((40, 10, 10), "mixed", CG, {"vel_tile_slices": 3}, 1, dict(warps_per_slice=2), dict(blocks_per_sm=2)),
])
def test_forms_of_the_partition_tests(monkeypatch, size, prec, kind, tuning, wide, vel, p):
    if wide:
        monkeypatch.setenv("PFEM2_MG_WIDE_MIN", "1")
    v, q = forms([spec(size)], prec, kind, tuning)
    assert subset(vel, v), v
    assert subset(p, q), q


def test_form_limits():
    """one cluster up to 300 items (slices x components)"""
    v, _ = forms([spec((79, 59))], "fp64", BICG)   # 4,800 rows: 150 slices
    assert v["cluster"] == 1 and v["blocks"] == 16
    v, _ = forms([spec((79, 60))], "fp64", BICG)   # 153 slices
    assert v["cluster"] == 0
    # 2D levels stay with the blocks' halo lists, restricted by groups of 8 lanes
    _, q = forms([spec((128, 48))], "fp64", CG)
    assert q["level1_published"] == 0 and q["restriction_lanes"] == 8


def test_forms_of_batches():
    """a block may hold parts of several instances"""
    v, q = forms([spec((23, 3)) for _ in range(1500)], "fp64", CG)
    assert v["systems_per_block"] > 10 and v["cluster"] == 0
    assert q["systems_per_block"] > 3
    v, q = forms([spec(z) for z in ((60, 20), (97, 33), (31, 8))], "mixed", CG)
    assert v["systems_per_block"] == 4 and q["systems_per_block"] >= 1


def test_solver_in_a_moving_context_without_hierarchy():
    sp = spec((4, 2))
    s = Solver(sp, moving_mesh=True, precision=A.PREC_FP64)
    v, q = s.solver_forms()
    s.close()
    assert v["blocks"] >= 1 and not any(q.values())
