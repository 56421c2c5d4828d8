"""The stage kernel of one warp per group of elements against the warp-specialised one, bit for bit: every
degree and precision, groups that do not fill, single elements, element ranges, forcing and filter."""
import ctypes as C

import numpy as np
import pytest

from wavedg_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


def _stage(s, stage, dt, F, acc, lo, hi):
    from wavedg_b200._lib import check, lib

    check(lib().wdg_rk4_stage_elems(s._h, stage, dt, 0.3, None if F is None else C.c_void_p(F.data_ptr()), 7.0,
                                    None if acc is None else C.c_void_p(acc.data_ptr()), 0.6, lo, hi), "stage")


@pytest.mark.parametrize("n", range(2, 10))
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("nx,ny", [(1, 1), (7, 5), (41, 23), (83, 61)])
def test_matches_warp_specialised(gpu_lib, n, precision, nx, ny):
    import torch

    import wavedg_b200 as W

    v, q = mg.uniform_rect(nx, -1.0, 1.0, ny, -0.7, 0.9)
    rng = np.random.default_rng(n)
    v, q = mg.scrambled(v + rng.uniform(-0.1 / max(nx, ny), 0.1 / max(nx, ny), size=v.shape), q, seed=n)
    mesh = W.Mesh2D.from_vertices(v, q)
    bc = rng.integers(0, 3, size=mesh.n_edges(1)).astype(np.int32)
    real = torch.float64 if precision == "fp64" else torch.float32
    nel, dt = nx * ny, 0.1 * mesh.min_h() / n**2
    cut = nel // 2 & ~3
    u = rng.standard_normal(3 * n * n * nel)
    F = torch.from_numpy(rng.standard_normal(u.size)).to("cuda", real)
    out = []
    for explicit in (False, True):
        s = W.WaveSystem(mesh, n, bc, precision=precision)
        if explicit:
            s.set_kernel(2)
        s.upload(u)
        acc = torch.from_numpy(u.copy()).cuda()
        for forced in (False, True):
            for stage in range(5):
                for lo, hi in ((0, cut), (cut, nel)):
                    _stage(s, stage, dt, F if forced else None, acc if forced and stage == 4 else None, lo, hi)
        out.append((s.download(), acc.cpu().numpy()))
    assert np.array_equal(out[0][0], out[1][0]) and not np.array_equal(out[0][0], u)
    assert np.array_equal(out[0][1], out[1][1]) and not np.array_equal(out[0][1], u)


@pytest.mark.parametrize("n", range(2, 10))
@pytest.mark.parametrize("nx,ny", [(1, 1), (7, 5), (83, 61)])
def test_operators(gpu_lib, n, nx, ny):
    """Operator launches against the tiled kernel.  Both sum 2 n + O(1) products a value in FP64, in different
    orders: 64 roundings of the largest value cover it (n <= 9)."""
    import wavedg_b200 as W

    v, q = mg.uniform_rect(nx, -1.0, 1.0, ny, -0.7, 0.9)
    rng = np.random.default_rng(n)
    v, q = mg.scrambled(v + rng.uniform(-0.1 / max(nx, ny), 0.1 / max(nx, ny), size=v.shape), q, seed=n)
    mesh = W.Mesh2D.from_vertices(v, q)
    bc = rng.integers(0, 3, size=mesh.n_edges(1)).astype(np.int32)
    basis = W.QuadratureRule.quadrature_rule(n, W.QuadratureRule.GaussLobatto)
    u = rng.standard_normal(3 * n * n * nx * ny)
    for op in (W.WaveEquation(mesh, basis, True), W.WaveBC(mesh, bc, basis, True)):
        out = []
        for family in (-1, 1):
            op.disc.set_kernel(family)
            du = 0.01 * u[::-1].copy()
            op.action(u, du)
            out.append(du)
        scale = max(np.abs(out[1]).max(), np.abs(u).max() / 2)
        assert np.abs(out[0] - out[1]).max() <= 64 * 2.0**-53 * scale
