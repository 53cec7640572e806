"""The mesh elasticity's stopping rule against the system assembled here in
numpy: the solve ends on, and reports, the residual b - K u of the displacement
it returns, and a tolerance below the rounding of that residual is met at the
rounding.
"""
import numpy as np
import pytest

from pfem2_b200 import _abi as A
from pfem2_b200 import cases
from pfem2_b200.solver import Solver

pytestmark = pytest.mark.gpu

FIXED, BODY, DISP = (1, 2, 4), 3, (0.0, 0.002)


def face_vertices(mesh, bid):
    out = np.zeros(mesh.n_vertices, bool)
    for f in range(4):
        on = mesh.face_bid[:, f] == bid
        for v in range(4):
            if ((v >> (f // 2)) & 1) == f % 2:
                out[mesh.cells[on, v]] = True
    return out


def element_matrices(mesh, lam, mu):
    """[n_cells, 4, 2, 4, 2]: vertex and component of the row, then of the column; QGauss(2)"""
    X, c = mesh.vertices, mesh.cells
    bit = np.array([[v & 1, v >> 1] for v in range(4)])
    g = 0.5 - 0.5 / np.sqrt(3.0)
    K = np.zeros((len(c), 4, 2, 4, 2))
    for p in [(a, b) for a in (g, 1.0 - g) for b in (g, 1.0 - g)]:
        f = np.where(bit == 1, p, 1.0 - np.array(p))
        s = 2.0 * bit - 1.0
        dN = np.stack([s[:, 0] * f[:, 1], s[:, 1] * f[:, 0]], 1)
        J = np.einsum("nva,vb->nab", X[c], dN)
        G = np.einsum("vb,nba->nva", dN, np.linalg.inv(J))
        w = 0.25 * np.linalg.det(J)
        K += lam * np.einsum("nia,njb,n->niajb", G, G, w) + mu * np.einsum("nib,nja,n->niajb", G, G, w)
        gg = mu * np.einsum("nic,njc,n->nij", G, G, w)
        for a in range(2):
            K[:, :, a, :, a] += gg
    return K


@pytest.mark.parametrize("cells,lam,rtol", [
    (2000, 1.0, 1e-12),
    (8200, 1.0, 1e-8),
    (8200, 1.0, 1e-12),
    (8200, 1.0, 1e-16),   # below the rounding of b - K u
    (30000, 1.0, 1e-16),  # a grid of blocks
    (2000, 100.0, 1e-12),
])
def test_residual_is_that_of_the_displacement(cells, lam, rtol):
    sp = cases.channel_disk(h=float(np.sqrt(4.0 / cells)))
    s = Solver(sp, precision=A.PREC_FP64, moving_mesh=True)
    it, res = s.problem_of_elasticity(lam, 1.0, FIXED, BODY, DISP, rtol=rtol)
    x = np.stack([s.field(A.FIELD_DISP_X), s.field(A.FIELD_DISP_Y)], 1)
    s.close()
    m = sp.mesh
    K = element_matrices(m, lam, 1.0)
    body = face_vertices(m, BODY)
    fix = body | np.any([face_vertices(m, b) for b in FIXED], axis=0)
    g = np.where(body[:, None], np.array(DISP), 0.0)
    assert np.array_equal(x[fix], g[fix])

    def product(Ke, v):
        out = np.zeros_like(v)
        np.add.at(out, m.cells, np.einsum("niajb,njb->nia", Ke, v[m.cells]))
        return out

    r = -product(K, x)[~fix]
    b = -product(K, np.where(fix[:, None], g, 0.0))
    diag = np.zeros_like(x)
    np.add.at(diag, m.cells, np.einsum("niaia->nia", K))
    b[fix] = (diag * g)[fix]
    true, tol = np.linalg.norm(r), rtol * np.linalg.norm(b)
    # what rounding each displacement and each product to FP64 leaves of b - K u
    # (independent errors; the element products bound the assembled ones)
    rounding = 2.0 ** -53 * np.sqrt(product(K * K, x * x)[~fix].sum())
    assert true <= max(tol, 8.0 * rounding)
    assert abs(res - true) <= 1e-3 * true + 8.0 * rounding
    assert it < 10000
