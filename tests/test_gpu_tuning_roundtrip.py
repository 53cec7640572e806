"""The launch shapes a context reports, given to another context of the same
instances, make it run the same kernels: the solvers add up their partial sums
in the partition's order, so that only the same partition gives the same bits.
"""
import numpy as np
import pytest

from pfem2_b200 import _abi as A
from pfem2_b200 import cases
from pfem2_b200.solver import Solver
from tests.test_gpu_parity import smooth_field

pytestmark = pytest.mark.gpu


def run(specs, tuning, **kw):
    s = Solver(specs, tuning=tuning, **kw)
    for i, sp in enumerate(specs):
        for d, v in enumerate(smooth_field(sp.mesh.vertices, 0.5)):
            s.set_field(A.FIELD_VX + d, v, i)
    s.seed_particles(specs[0].q, 0, 0.1)
    for _ in range(2):
        s.step()
    s.stats()
    out = [s.field(f, i) for i in range(len(specs)) for f in (A.FIELD_VX, A.FIELD_VY, A.FIELD_P)]
    t = s.tuning()
    s.close()
    return t, out


@pytest.mark.parametrize("sizes,prec,kind", [
    ([(32, 12)], A.PREC_FP64, A.SOLVER_BICGSTAB),            # one cluster
    ([(64, 16)], A.PREC_MIXED, A.SOLVER_CG),                 # one cluster
    ([(128, 48)], A.PREC_FP64, A.SOLVER_BICGSTAB),           # a grid, two blocks per SM
    ([(317, 101)], A.PREC_MIXED, A.SOLVER_BICGSTAB),         # a grid, one block per SM
    ([(60, 20), (97, 33), (31, 8)], A.PREC_FP64, A.SOLVER_CG),  # a batch
    ([(128, 96)] * 24, A.PREC_MIXED, A.SOLVER_CG),           # a batch larger than the grid's least slices
])
def test_reported_shapes_reproduce_the_run(sizes, prec, kind):
    specs = []
    for nx, ny in sizes:
        sp = cases.poiseuille_2d(nx=nx, ny=ny)
        sp.case.vel_solver = kind
        sp.case.vel_tol = sp.case.p_tol = 0.0
        sp.case.vel_rtol = sp.case.p_rtol = 1e-9
        specs.append(sp)
    t, a = run(specs, None, precision=prec)
    t2, b = run(specs, t, precision=prec)
    assert t2 == t
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("end,advect,vel", [
    ("1.2345", 16, 0),      # written for the kernels before: automatic shapes
    ("1.2345 v2", 3, 7),
])
def test_cache_lines_of_former_kernels_are_passed_over(tmp_path, monkeypatch, end, advect, vel):
    sp = cases.poiseuille_2d(nx=32, ny=12)
    s = Solver(sp, precision=A.PREC_FP64)
    key = s.tuning_key()
    s.close()
    path = tmp_path / "tuning.txt"
    path.write_text(f"{key} 3 1 2 7 1 1 {end}\n")
    monkeypatch.setenv("PFEM2_TUNING_CACHE", str(path))
    s = Solver(sp, precision=A.PREC_FP64)
    t = s.tuning()
    s.close()
    assert t["advect_blocks_per_sm"] == advect and t["vel_tile_slices"] == vel
