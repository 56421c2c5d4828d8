"""A handle's device memory is complete after its first upload (or array step): nothing that a
WaveHoltz period or a captured step launches later allocates, whichever of the resident and the
streaming kernels it takes.  The meshes and CTA limits stand on both sides of what fits the chip:
the FP32 mesh is resident without forcing only, the limits leave none or some of the launches resident."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(nx, n, precision, cap=0, kernel=None):
    import wavedg_b200 as W

    s = W.WaveSystem(W.Mesh2D.uniform_rect(nx, -1.0, 1.0, nx, -1.0, 1.0), n, None, precision=precision)
    if cap:
        s.set_max_ctas(cap)
    if kernel is not None:
        s.set_kernel(kernel)
    return s


@pytest.mark.parametrize("nx,n,precision,cap,omega", [(120, 8, "fp32", 0, 200.0), (191, 5, "fp32", 0, 200.0),
                                                      (64, 5, "fp64", 20, 60.0), (64, 5, "fp64", 48, 60.0),
                                                      (40, 7, "fp32", 9, 60.0), (24, 4, "fp64", 1, 30.0)])
def test_waveholtz_on_a_fresh_handle(gpu_lib, nx, n, precision, cap, omega):
    import wavedg_b200 as W

    got = []
    for s in (_system(nx, n, precision, cap), _system(nx, n, precision, 0, 2)):
        F = np.random.default_rng(7).standard_normal(s.ndof)
        wh = W.WaveHoltz(omega, s.mesh, n, None, True, system=s)
        w = np.zeros(s.ndof)
        wh.pi0(w, F)
        x = w.copy()
        wh.S(x)
        got.append((w, x))
    # the filter's FP64 sums of at most 250 steps round in another order; FP64 adds the forcing elsewhere
    for x, y in zip(*got):
        assert np.linalg.norm(x - y) <= 1e-12 * np.linalg.norm(y)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("nx,change", [(19, None), (19, "kernel"), (19, "cap"), (64, "cap"), (260, None)])
def test_first_step_is_captured(gpu_lib, precision, nx, change):
    import torch

    a, b = _system(nx, 5, precision), _system(nx, 5, precision, 0, 2)
    u = np.random.default_rng(1).standard_normal(a.ndof)
    dt = 0.1 * a.mesh.min_h() / 25
    a.upload(u)
    b.upload(u)
    if change:
        a.step_state(dt, 0.0, 1)
        b.step_state(dt, 0.0, 1)
    if change == "kernel":
        a.set_kernel(2)
    if change == "cap":
        a.set_max_ctas(3)
    a.sync()
    stream = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        a.set_stream(stream)
        with torch.cuda.graph(graph, stream=stream):
            a.step_state(dt, 0.0, 2)
        graph.replay()
        a.set_kernel(-1)
        a.step_state(dt, 0.0, 1)  # the first launch outside a graph, behind a replay
        graph.replay()
    stream.synchronize()
    b.step_state(dt, 0.0, 5)
    assert np.array_equal(a.download(), b.download())


def test_steps_do_not_allocate(gpu_lib):
    import torch

    s = _system(128, 5, "fp64")
    s.upload(np.zeros(s.ndof))
    s.step_state(0.0, 0.0, 0)
    _system(16, 5, "fp64").rk4_steps(np.zeros(3 * 25 * 256), 0.0, 0.0, 1)  # the kernels are loaded
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    s.step_state(1e-4, 0.0, 2)
    s.set_kernel(2)
    s.step_state(1e-4, 0.0, 2)
    s.sync()
    assert torch.cuda.mem_get_info()[0] == free


@pytest.mark.parametrize("precision,nx", [("fp64", 32), ("fp64", 200)])
def test_array_steps_hold_no_state(gpu_lib, precision, nx):
    """Steps on the caller's array allocate what steps work in and no state; the state comes with its upload,
    and both then give the same."""
    import torch

    import wavedg_b200 as W

    s = _system(nx, 4, precision)
    u = torch.randn(s.ndof, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    x = u.clone()
    dt = 0.1 * s.mesh.min_h() / 16
    s.rk4_steps(x, dt, 0.0, 2)
    with pytest.raises(W.WdgError):
        s.step_state(dt, 0.0, 1)
    s.upload(u)
    s.step_state(dt, 0.0, 2)
    assert np.array_equal(s.download(), x.cpu().numpy())
