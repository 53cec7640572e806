"""Move and re-sort of a mesh whose counts take the scan's look-back over more
than 32 tiles of 2,048 cells (one window of it), against the oracle.
"""
import numpy as np
import pytest

from pfem2_b200 import _abi as A
from pfem2_b200 import cases
from tests.test_gpu_parity import XI_TOL, make_pair, set_vel, smooth_field

pytestmark = pytest.mark.gpu


def test_scan_over_many_tiles():
    sp = cases.poiseuille_2d(nx=540, ny=131)  # 70,740 cells: 35 tiles, the last one ragged
    sp.case.dt = 0.005
    g, o = make_pair(sp, "fp64", particles_only=True)
    set_vel(g, o, sp, smooth_field(sp.mesh.vertices))
    g.seed_particles((2, 2), seed=5, jitter=0.1)
    o.seed_particles((2, 2), seed=5, jitter=0.1)
    for _ in range(2):
        g.move_particles()
        o.move_particles()
    cg, xg, ug = g.particles()
    co, xo, uo = o.particles()
    assert np.array_equal(cg, co)
    assert np.abs(xg - xo).max() <= XI_TOL["fp64"]
    assert np.abs(ug - uo).max() <= 1e-12 * max(1.0, np.abs(uo).max())
    gs, os_ = g.stats(), o.stats()
    for k in ("deleted", "removed", "reseeded"):
        assert gs[k] == os_[k]
