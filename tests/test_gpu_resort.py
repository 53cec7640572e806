"""Move and re-sort at the sizes where its lists change form, against the
oracle (which moves one particle at a time, TurekBenchmark/pfem2particle.cpp):
few and many particles per cell (lists up to the stored 64 entries and beyond),
up to 32 sub-cells (a mask) and more (counts), one and several chunks of 32
particles, cells that receive more movers than their mover list holds, and
movers beyond the 1-ring. FP64 particles: same cells in the same storage order,
coordinates and velocities to rounding (the bars of the parity tests).
"""
import numpy as np
import pytest

from pfem2_b200 import _abi as A
from tests.test_gpu_parity import XI_TOL, make_pair, set_vel, smooth_field, spec_2d, spec_3d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,q,scale,crowd", [
    (2, (1, 1), 1.0, 0),        # one particle a cell
    (2, (2, 3), 1.0, 100),      # mover list of 32, a hundred movers at once
    (2, (6, 6), 1.0, 0),        # 36 sub-cells: counts, two chunks
    (2, (9, 9), 1.0, 300),      # lists beyond the stored length
    (2, (4, 8), 4.0, 0),        # 32 sub-cells: the mask's last bit; far movers
    (3, (3, 3, 3), 1.0, 90),    # mover list of 64
    (3, (4, 4, 5), 1.0, 0),     # 80 sub-cells
])
def test_resort(dim, q, scale, crowd):
    sp = spec_2d() if dim == 2 else spec_3d()
    g, o = make_pair(sp, "fp64")
    f = smooth_field(sp.mesh.vertices, scale)
    set_vel(g, o, sp, f)
    g.seed_particles(q, seed=5, jitter=0.1)
    o.seed_particles(q, seed=5, jitter=0.1)
    cell, xi, u = g.particles()
    if crowd:
        # `crowd` more particles near the outflow side of an inner cell
        c = sp.mesh.n_cells // 2 + 3
        rng = np.random.default_rng(3)
        x = rng.random((crowd, dim))
        x[:, 0] = 0.95 + 0.04 * x[:, 0]
        k = np.searchsorted(cell, c, side="right")
        cell = np.insert(cell, k, np.full(crowd, c, cell.dtype))
        xi = np.insert(xi, k, x, axis=0)
        u = np.insert(u, k, rng.standard_normal((crowd, dim)), axis=0)
        g.set_particles([(cell, xi, u)])
        o.set_particles(cell, xi, u)
    far = 0
    for step in range(3):
        if step == 1 or (crowd and step == 0):
            g.advect()
            o.advect()
        else:
            g.move_particles()
            o.move_particles()
        far += g.stats()["far"]
    cg, xg, ug = g.particles()
    co, xo, uo = o.particles()
    assert np.array_equal(cg, co)
    assert np.abs(xg - xo).max() <= XI_TOL["fp64"]
    assert np.abs(ug - uo).max() <= 1e-12 * max(1.0, np.abs(uo).max())
    assert (far > 0) == (scale > 1.0)
    gs, os_ = g.stats(), o.stats()
    for k in ("deleted", "removed", "reseeded"):
        assert gs[k] == os_[k]


@pytest.mark.parametrize("dim,q,scale,blocks,prec", [
    (2, (1, 1), 1.0, 32, "fp64"),   # chunks of a few particles, units of one
    (2, (5, 5), 1.0, 1, "fp64"),    # several slices a warp, full units
    (2, (5, 5), 4.0, 4, "fp32"),    # far movers, FP32 storage
    (3, (3, 3, 3), 1.0, 2, "fp64"),
    (3, (2, 2, 2), 1.0, 32, "fp32"),
])
def test_advection_forms(dim, q, scale, blocks, prec):
    """the two-kernel advection moves every particle bit for bit as the
    one-kernel form does, for chunks from below a warp to many slices"""
    out = []
    for split in (1, 2):
        sp = spec_2d() if dim == 2 else spec_3d()
        g, o = make_pair(sp, prec, tuning={"advect_split": split, "advect_blocks_per_sm": blocks})
        set_vel(g, o, sp, smooth_field(sp.mesh.vertices, scale))
        g.seed_particles(q, seed=5, jitter=0.1)
        for _ in range(3):
            g.advect()
        out.append((g.particles(), g.stats()["deleted"], g.stats()["far"]))
    (a, da, fa), (b, db, fb) = out
    assert da == db and fa == fb
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
