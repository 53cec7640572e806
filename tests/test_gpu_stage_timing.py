"""Stage timing of steps with and without a CUDA graph, and of contexts that
call the FEM step by itself.
"""
import numpy as np
import pytest

from pfem2_b200 import _abi as A
from pfem2_b200.solver import Solver
from tests.test_gpu_parity import spec_2d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_graph", [True, False])
def test_stage_times(use_graph):
    sp = spec_2d(dt=0.01)
    s = Solver(sp, precision=A.PREC_FP64, use_graph=use_graph)
    s.seed_particles(sp.q, 0, 0.1)
    s.enable_stage_timing(True)
    s.step()
    s.step()
    assert (s.stage_times(reset=True) > 0.0).all()
    s.correct_particles_velocities()
    s.move_particles()
    s.distribute_particle_velocities_to_grid()
    s.fem_step()  # not a timed step
    assert not np.any(s.stage_times(reset=True))
    s.step()
    assert (s.stage_times() > 0.0).all()
    s.close()
