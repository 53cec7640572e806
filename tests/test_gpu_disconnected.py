"""The pressure hierarchy of a large mesh with a small part by itself."""
import resource

import numpy as np
import pytest

from pfem2_b200 import _abi as A
from pfem2_b200 import cases
from pfem2_b200 import meshes as M
from pfem2_b200.solver import Pfem2Error, Solver

pytestmark = pytest.mark.gpu


def joined(a, b):
    return M.Mesh(np.concatenate([a.vertices, b.vertices]),
                  np.concatenate([a.cells, b.cells + a.n_vertices]).astype(a.cells.dtype),
                  np.concatenate([a.face_bid, b.face_bid]))


def test_level_two_is_coarsened_beside_a_small_part():
    """level 2 is stored as a dense matrix and coarsened to at most 6,144
    unknowns; a 6 x 6 part that has come down to one unknown stays as it is"""
    sp = cases.poiseuille_2d(nx=1600, ny=400)
    alone = Solver(sp, precision=A.PREC_MIXED)
    n_alone = alone.solver_sizes()
    alone.close()
    sp.mesh = joined(sp.mesh, M.rect_mesh(6, 6, 5.0, 6.0, 0.0, 1.0))
    s = Solver(sp, precision=A.PREC_MIXED)
    n = s.solver_sizes()
    s.close()
    assert n_alone["n2"] <= 6144 and n["n2"] <= 6144
    assert n_alone["n2"] < n["n2"] <= n_alone["n2"] + 4


def test_solution_beside_a_small_part():
    """The flow of the channel does not change with the part beside it. The
    smallest eigenvalue of the pressure matrix, (pi / 8)^2 / 24^2, turns a residual
    of 1e-12 on either side into 7e-9 of P, and the correction, dt / h = 1.2 times
    its differences, into less than 1e-7 of V."""
    out = []
    for part in (False, True):
        sp = cases.poiseuille_2d(nx=96, ny=24)
        if part:
            sp.mesh = joined(sp.mesh, M.rect_mesh(6, 6, 5.0, 6.0, 0.0, 1.0))
        sp.case.dt = 0.05
        sp.case.vel_tol = sp.case.p_tol = 1e-12
        s = Solver(sp, precision=A.PREC_FP64)
        X = sp.mesh.vertices
        s.set_field(A.FIELD_VX, np.where(X[:, 0] <= 4.0, 4.0 * X[:, 1] * (1.0 - X[:, 1]), 0.0))
        s.fem_step()
        s.stats()
        out.append([s.field(f)[:97 * 25] for f in (A.FIELD_VX, A.FIELD_VY, A.FIELD_P)])
        s.close()
    for x, y in zip(*out):
        assert np.linalg.norm(x - y) <= 1e-7 * max(1.0, np.linalg.norm(x))


def test_more_parts_than_a_block_holds_is_refused():
    """each of 30,000 parts has a level-2 unknown at least, 240 KB in FP64: the
    refusal comes before a dense matrix of that size (7.2 GB) is made, and
    leaves the process able to make another context"""
    part = M.rect_mesh(5, 5)
    k = 30000
    sp = cases.poiseuille_2d(nx=4, ny=2)
    shift = np.stack([2.0 * (np.arange(k) % 200), 2.0 * (np.arange(k) // 200)], 1)
    nv = part.n_vertices
    sp.mesh = M.Mesh((part.vertices[None] + shift[:, None]).reshape(-1, 2),
                     (part.cells[None] + nv * np.arange(k)[:, None, None]).reshape(-1, 4).astype(part.cells.dtype),
                     np.tile(part.face_bid, (k, 1)))
    before = resource.getrusage(resource.RUSAGE_SELF).ru_maxrss
    with pytest.raises(Pfem2Error) as e:
        Solver(sp, precision=A.PREC_FP64)
    assert e.value.status == A.INVALID_ARG and "shared memory" in str(e.value)
    assert resource.getrusage(resource.RUSAGE_SELF).ru_maxrss - before < 5_000_000  # kB
    s = Solver(cases.poiseuille_2d(nx=32, ny=12), precision=A.PREC_FP64)
    s.close()
