"""Which advection runs: one kernel for small sets of particles in 2D, two
otherwise, by the particles of the last seeding; the environment variable and
the launch shapes override the rule. Both forms move every particle bit for bit
alike (tests/test_gpu_resort.py).
"""
import numpy as np
import pytest

from pfem2_b200 import _abi as A
from pfem2_b200 import cases
from pfem2_b200.solver import Solver

pytestmark = pytest.mark.gpu


def split(s):
    return s.tuning()["advect_split"]


@pytest.mark.parametrize("dim,size,q,want", [
    (2, (32, 12), (4, 4), 1),
    (2, (128, 64), (4, 4), 2),      # 131,072 particles
    (2, (127, 64), (4, 4), 1),
    (3, (12, 6, 6), (1, 1, 1), 2),
])
def test_rule(monkeypatch, dim, size, q, want):
    sp = cases.poiseuille_2d(nx=size[0], ny=size[1]) if dim == 2 else cases.pipe_3d(nx=size[0], ny=size[1], nz=size[2])
    s = Solver(sp, precision=A.PREC_FP64, particles_only=True, capacity_factor=4.0)
    s.seed_particles(q, 0, 0.1)
    assert split(s) == want
    s.step()
    a = s.particles()
    s.close()
    for v in (1, 2):
        s = Solver(sp, precision=A.PREC_FP64, particles_only=True, capacity_factor=4.0, tuning={"advect_split": v})
        s.seed_particles(q, 0, 0.1)
        assert split(s) == v
        s.step()
        for x, y in zip(s.particles(), a):
            assert np.array_equal(x, y)
        s.close()
    monkeypatch.setenv("PFEM2_ADVECT_SPLIT_MIN", "0")
    s = Solver(sp, precision=A.PREC_FP64, particles_only=True)
    s.seed_particles(q, 0, 0.1)
    assert split(s) == 2
    s.close()


def test_rule_follows_the_last_seeding():
    sp = cases.poiseuille_2d(nx=128, ny=64)
    s = Solver(sp, precision=A.PREC_FP64, particles_only=True)
    s.seed_particles((4, 4), 0, 0.1)
    assert split(s) == 2
    s.step()
    s.seed_particles((2, 2), 0, 0.1)
    assert split(s) == 1
    s.step()
    s.close()
