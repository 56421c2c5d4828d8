"""The fused exact-quadrature kernel at every degree, for each of its models, on meshes whose element
counts leave partial groups, against the plain FP64 torch restatement in perf/cases.py (with Gauss
rules polished in extended precision: numpy's weights are 1e-14 off at 18 points, which the inverse
mass matrix of degree 8 raises to 1e-11 in a nearly uniform gas).

Tolerance 1e-12 (relative 2-norm), the suite's bound per right-hand side: both sides sum at most a
few thousand FP64 terms of like size, about 1e-14."""
import importlib.util
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cases():
    path = os.path.join(os.path.dirname(__file__), "..", "perf", "cases.py")
    spec = importlib.util.spec_from_file_location("perf_cases", path)
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    m._legendre = _gauss
    return m


def _gauss(n):
    x = np.polynomial.legendre.leggauss(n)[0].astype(np.longdouble)
    for _ in range(4):
        p0, p1 = np.ones_like(x), x.copy()
        for k in range(2, n + 1):
            p0, p1 = p1, ((2 * k - 1) * x * p1 - (k - 1) * p0) / k
        dp = n * (x * p1 - p0) / (x * x - 1)
        x = x - p1 / dp
    return x.astype(np.float64), (2 / ((1 - x * x) * dp * dp)).astype(np.float64)


@pytest.mark.parametrize("n", range(2, 10))
@pytest.mark.parametrize("kind", ["wave", "euler", "advect-gll", "advect-gl"])
def test_exact_rhs(gpu_lib, kind, n):
    import torch

    M = _cases()
    nx, ny = (7, 5) if n % 2 else (3, 11)
    case = dict(kind={"wave": "exactq", "euler": "euler"}.get(kind, "vadvect"), nx=nx, ny=ny, n=n, mesh="scrambled",
                bc="mixed", approx=False, legendre=kind == "advect-gl")
    _, _, d = M._disc(case, n)
    u = M._state(case, d, n)
    s = M.prepare(dict(case, steps=1, method="rk4"), n)["sys"]
    out = torch.zeros(u.numel(), dtype=torch.float64, device="cuda")
    s.rhs(u.reshape(-1).contiguous(), out)
    if kind == "wave":
        rhs = M._wave_rhs(d, M._side_codes(d, "mixed"))
    elif kind == "euler":
        rhs = M._euler_rhs(d)
    else:
        rhs = M._vadvect_rhs(d, M._rotation(d))
    ref = rhs(u).reshape(-1)
    assert float((out - ref).norm() / ref.norm()) < 1e-12
    if kind == "wave":
        F = torch.from_numpy(np.random.default_rng(n).standard_normal(u.numel())).to("cuda")
        s.rhs(u.reshape(-1).contiguous(), out, F, 0.7)
        ref = ref + 0.7 * d.inv_mass(F.reshape(u.shape)).reshape(-1)
        assert float((out - ref).norm() / ref.norm()) < 1e-12
