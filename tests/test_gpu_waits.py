"""Bounded waits that run out, in each kernel an RK4 call can take: flags of a neighbouring group that
never come (resident steps, alone and in a batch), a group or chunk that is never loaded (one warp per
CTA, warp-specialised).  Nothing faults: a host-set hook leaves the work out, the kernels give up after
the handle's limit and return, the call reports it, and the handle's next step is right."""
import ctypes as C
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(nx, n, precision, explicit=False):
    import wavedg_b200 as W

    s = W.WaveSystem(W.Mesh2D.uniform_rect(nx, -1.0, 1.0, nx, -1.0, 1.0), n, None, precision=precision)
    if explicit:
        s.set_kernel(2)
    return s


def _resident(s):
    import wavedg_b200 as W

    n = C.c_int(-1)
    assert W.lib().wdg_test_resident(s._h, 0, C.byref(n)) == 0
    return n.value > 0


# the last two columns: whether the mesh is resident; the group or chunk left out
@pytest.mark.parametrize("nx,n,precision,explicit,resident,skip",
                         [(48, 5, "fp64", False, True, 0), (48, 5, "fp64", False, True, 383), (41, 8, "fp32", False, True, 200),
                          (5, 4, "fp64", False, True, 3), (160, 5, "fp64", False, False, 0), (160, 5, "fp64", False, False, 1),
                          (210, 5, "fp32", False, False, 1), (48, 5, "fp64", True, False, 0), (48, 6, "fp32", True, False, 0)])
def test_wait_runs_out(gpu_lib, nx, n, precision, explicit, resident, skip):
    import wavedg_b200 as W

    L = W.lib()
    s = _system(nx, n, precision, explicit)
    assert _resident(s) == resident
    u0 = np.random.default_rng(nx).standard_normal(s.ndof)
    dt = 0.1 * s.mesh.min_h() / n**2
    want = u0.copy()
    _system(nx, n, precision, explicit).rk4_steps(want, dt, 0.0, 2)
    assert L.wdg_wave_set_wait_limit(s._h, 0.005) == 0
    assert L.wdg_test_skip_chunk(s._h, skip) == 0
    t0 = time.perf_counter()
    with pytest.raises(W.WdgError) as e:
        s.rk4_steps(u0.copy(), dt, 0.0, 2)
    took = time.perf_counter() - t0
    assert e.value.code == W._lib.WDG_ERR_TIMEOUT and "bounded device-side wait" in str(e.value)
    assert took < 1.0, took  # the limit, not the default of 2 s
    assert L.wdg_wave_set_wait_limit(s._h, 2.0) == 0
    for _ in range(2):
        u = u0.copy()
        s.rk4_steps(u, dt, 0.0, 2)
        np.testing.assert_array_equal(u, want)


def test_batch_reports_a_solve_whose_wait_ran_out(gpu_lib):
    import wavedg_b200 as W

    L = W.lib()
    systems = [_system(m, n, "fp64") for m, n in ((20, 5), (16, 4), (9, 7))]
    b = W.WaveHoltzBatch(systems, [5.0, 6.0, 7.0])
    F = [np.random.default_rng(k).standard_normal(s.ndof) for k, s in enumerate(systems)]
    want = b.solve(F, tol=1e-12, maxit=2)[0]
    for s in systems[:2]:
        assert L.wdg_wave_set_wait_limit(s._h, 0.005) == 0
        assert L.wdg_test_skip_chunk(s._h, 1) == 0
    with pytest.raises(W.WdgError) as e:
        b.solve(F, tol=1e-12, maxit=2)
    assert e.value.code == W._lib.WDG_ERR_TIMEOUT
    for s in systems:
        assert L.wdg_wave_set_wait_limit(s._h, 2.0) == 0
    got = b.solve(F, tol=1e-12, maxit=2)[0]  # nothing of either solve's error is left
    for x, y in zip(got, want):
        assert np.array_equal(x, y)
