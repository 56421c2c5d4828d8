"""The exact mass matrix and its inverse at every degree and basis, for one to many variables (fewer
elements per warp where their staging fills shared memory), on element counts that end inside a
group, in place and not, against the element matrices of the (n + 1)-point rule formed in numpy.

Tolerance 1e-13 for M x, 1e-12 for M^{-1} x, as for the golden vectors."""
import numpy as np
import pytest

from conftest import rel
from wavedg_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


def _matrices(mesh_v, mesh_q, x):
    n = len(x)
    g, w = np.polynomial.legendre.leggauss(n + 1)
    L = np.array([[np.prod([(p - x[m]) / (x[k] - x[m]) for m in range(n) if m != k]) for k in range(n)] for p in g])
    phi = np.einsum("pi,qj->qpji", L, L).reshape((n + 1) ** 2, n * n)  # points (eta, xi), nodes (j, i)
    c = mesh_v[mesh_q]  # (elements, corner, xy)
    xi, eta = g[None, :, None], g[:, None, None]
    Jx = 0.25 * ((1 - eta) * (c[:, None, None, 1] - c[:, None, None, 0]) + (1 + eta) * (c[:, None, None, 2] - c[:, None, None, 3]))
    Je = 0.25 * ((1 - xi) * (c[:, None, None, 3] - c[:, None, None, 0]) + (1 + xi) * (c[:, None, None, 2] - c[:, None, None, 1]))
    det = Jx[..., 0] * Je[..., 1] - Jx[..., 1] * Je[..., 0]
    wd = (det * w[None, :, None] * w[None, None, :]).reshape(len(mesh_q), -1)
    return np.einsum("pa,ep,pb->eab", phi, wd, phi)


@pytest.mark.parametrize("n", range(2, 10))
@pytest.mark.parametrize("gauss", ["GaussLobatto", "GaussLegendre"])
@pytest.mark.parametrize("nv,nx", [(1, 5), (3, 9), (2, 1), (18, 3)])
def test_action_and_inverse(gpu_lib, n, gauss, nv, nx):
    import wavedg_b200 as W

    v, q = mg.perturbed_rect(nx, 0.2, seed=n) if nx > 1 else mg.uniform_rect(1, -1.0, 0.3, 1, -0.5, 1.0)
    mesh = W.Mesh2D.from_vertices(v, q)
    rule = W.QuadratureRule.quadrature_rule(n, getattr(W.QuadratureRule, gauss))
    M = _matrices(np.asarray(v), np.asarray(q), np.asarray(rule.x))
    x = np.random.default_rng(nv).standard_normal((len(q), n * n, nv))
    m = W.BasisMassMatrix(mesh, rule, False)
    y = np.zeros(x.size)
    m.action(nv, x.reshape(-1), y)
    assert rel(y, np.einsum("eab,ebd->ead", M, x)) < 1e-13
    z = x.reshape(-1).copy()
    m.inv(nv, z)
    assert rel(z, np.linalg.solve(M, x)) < 1e-12
