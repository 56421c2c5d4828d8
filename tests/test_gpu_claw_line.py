"""The fused collocation kernel of the conservation laws at every degree and variable count, with
partial groups, on 16-byte aligned arrays (bulk copies) and on arrays 8 bytes off (plain copies),
against the plain FP64 torch restatement in perf/cases.py.

Tolerance 1e-12 (relative 2-norm), the suite's bound per right-hand side."""
import importlib.util
import os

import pytest

pytestmark = pytest.mark.gpu


def _cases():
    path = os.path.join(os.path.dirname(__file__), "..", "perf", "cases.py")
    spec = importlib.util.spec_from_file_location("perf_cases", path)
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


def _check(kind, n, nv, shift):
    import torch

    M = _cases()
    nx, ny = (7, 5) if n % 2 else (3, 11)
    case = dict(kind=kind, nx=nx, ny=ny, n=n, nv=nv, mesh="scrambled", approx=True, steps=1, method="rk4")
    _, _, d = M._disc(case, n)
    u = M._state(case, d, n)
    s = M.prepare(case, n)["sys"]
    buf = torch.zeros(2, u.numel() + 2, dtype=torch.float64, device="cuda")
    x, out = buf[0, shift:shift + u.numel()], buf[1, shift:shift + u.numel()]
    x.copy_(u.reshape(-1))
    rhs = M._euler_rhs(d) if kind == "euler" else M._advect_rhs(d, M._t(M._matrices(nv, n)))
    ref = rhs(u).reshape(-1)
    s.rhs(x, out)
    assert float((out - ref).norm() / ref.norm()) < 1e-12
    # a step of every stage form, large enough to show in the state
    dt = 1e-3
    if kind == "euler":
        for method in ("ssprk3", "rk4"):
            x.copy_(u.reshape(-1))
            s.steps(x, dt, 0.0, 2, method)
            ref = M._advance(rhs, u, dt, 2, method).reshape(-1)
            assert float((x - ref).norm() / (ref - u.reshape(-1)).norm()) < 1e-12
        # the volume term alone is added to the output
        out.fill_(2.0)
        s.div(u.reshape(-1).contiguous() if shift == 0 else x.copy_(u.reshape(-1)), out)
        q = u
        rho, mx, my, E = q.unbind(-1)
        a, b = mx / rho, my / rho
        p = 0.4 * (E - 0.5 * rho * (a * a + b * b))
        ref = 2.0 + d.volume(torch.stack([mx, mx * a + p, mx * b, a * (E + p)], -1),
                             torch.stack([my, mx * b, my * b + p, b * (E + p)], -1)).reshape(-1)
        assert float((out - ref).norm() / ref.norm()) < 1e-12
    else:
        x.copy_(u.reshape(-1))
        s.rk4_steps(x, dt, 0.0, 2)
        ref = M._advance(rhs, u, dt, 2).reshape(-1)
        assert float((x - ref).norm() / (ref - u.reshape(-1)).norm()) < 1e-12


@pytest.mark.parametrize("n", range(2, 10))
@pytest.mark.parametrize("shift", [0, 1])
def test_euler(gpu_lib, n, shift):
    _check("euler", n, 4, shift)


@pytest.mark.parametrize("n,nv", [(2, 1), (2, 8), (3, 3), (4, 5), (5, 1), (5, 2), (5, 7), (6, 4), (7, 6), (8, 2), (9, 3), (9, 8)])
@pytest.mark.parametrize("shift", [0, 1])
def test_linear(gpu_lib, n, nv, shift):
    _check("advect", n, nv, shift)
