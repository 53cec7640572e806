"""A refused pfem2_set_particles leaves the particles as they are, also after a
read, which packs what it copies into the idle half of the particle storage.
"""
import numpy as np
import pytest

from pfem2_b200 import _abi as A
from pfem2_b200.solver import Pfem2Error, Solver
from tests.test_gpu_parity import smooth_field, spec_2d

pytestmark = pytest.mark.gpu


def context(stages, steps):
    sp = spec_2d(dt=0.01)
    s = Solver(sp, precision=A.PREC_MIXED, fp32_stages=stages)
    for d, v in enumerate(smooth_field(sp.mesh.vertices, 0.5)):
        s.set_field(A.FIELD_VX + d, v)
    s.seed_particles((4, 4), 0, 0.1)
    for _ in range(steps):
        s.step()
    return s


@pytest.mark.parametrize("stages", [0, A.FP32_ALL])
@pytest.mark.parametrize("steps", [1, 2])
@pytest.mark.parametrize("bad", ["value", "cell", "more"])
def test_refused_set_particles_changes_nothing(stages, steps, bad):
    a, b = context(stages, steps), context(stages, steps)
    want = b.particles()
    cell, xi, u = [x.copy() for x in a.particles()]
    if bad == "more":  # more than the storage holds, refused for a value at the end
        cell, xi, u = np.tile(cell, 5), np.tile(xi, (5, 1)), np.tile(u, (5, 1))
    if bad == "cell":
        cell[-1] = a.specs[0].mesh.n_cells
    else:
        u[-1, 0] = np.nan
    with pytest.raises(Pfem2Error) as e:
        a.set_particles([(cell, xi, u)])
    assert e.value.status == A.INVALID_ARG
    for x, y in zip(a.particles(), want):
        assert np.array_equal(x, y)
    a.step()
    b.step()
    for x, y in zip(a.particles(), b.particles()):
        assert np.array_equal(x, y)
    a.close()
    b.close()
