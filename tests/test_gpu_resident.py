"""The resident RK4 launch (elements on chip for all steps) against the streaming stage kernel, bit for
bit: every degree and precision, from one element to several rounds of groups per warp, under CTA
caps, inside captured graphs replayed between eager calls, and with WaveHoltz's forcing and filter."""
import numpy as np
import pytest

from wavedg_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


def _pair(nx, ny, n, precision, seed):
    import wavedg_b200 as W

    v, q = mg.uniform_rect(nx, -1.0, 1.0, ny, -0.7, 0.9)
    rng = np.random.default_rng(seed)
    v = v + rng.uniform(-0.1 / max(nx, ny), 0.1 / max(nx, ny), size=v.shape)
    v, q = mg.scrambled(v, q, seed=seed)
    mesh = W.Mesh2D.from_vertices(v, q)
    bc = rng.integers(0, 3, size=mesh.n_edges(1)).astype(np.int32)
    a, b = (W.WaveSystem(mesh, n, bc, precision=precision) for _ in range(2))
    b.set_kernel(2)  # an explicit choice: the streaming kernel
    return a, b, rng.standard_normal(a.ndof), 0.1 * mesh.min_h() / n**2


@pytest.mark.parametrize("n", range(2, 10))
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("nx,ny,cap", [(1, 1, 0), (7, 5, 0), (41, 23, 0), (17, 9, 3)])
def test_matches_streaming(gpu_lib, n, precision, nx, ny, cap):
    a, b, u, dt = _pair(nx, ny, n, precision, n)
    a.set_max_ctas(cap)
    x, y = u.copy(), u.copy()
    for steps in (1, 3):  # the second launch counts on from the first one's flags
        ta, tb = a.rk4_steps(x, dt, 0.0, steps), b.rk4_steps(y, dt, 0.0, steps)
        assert ta == tb
        assert np.array_equal(x, y)
    assert not np.array_equal(x, u)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_captured(gpu_lib, precision):
    import torch

    a, b, u, dt = _pair(19, 13, 5, precision, 3)
    a.upload(u)
    b.upload(u)
    a.step_state(dt, 0.0, 2)
    stream = torch.cuda.Stream()
    a.sync()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        a.set_stream(stream)
        with torch.cuda.graph(graph, stream=stream):
            a.step_state(dt, 0.0, 2)
        for k in range(3):
            graph.replay()
            a.step_state(dt, 0.0, 1 + k)
    stream.synchronize()
    b.step_state(dt, 0.0, 2 + 3 * 2 + 6)
    assert np.array_equal(a.download(), b.download())


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_batch(gpu_lib, precision):
    """Batched solves as resident periods against the streaming launches (an explicit launch shape): uneven
    meshes, degrees and frequencies, more least shares than SMs, cold, warm and with a known |pi0|."""
    import wavedg_b200 as W
    from wavedg_b200.dg import WaveHoltzBatch

    rng = np.random.default_rng(11)
    shapes = [(9, 4), (31, 5), (8, 7), (5, 2), (24, 9), (40, 3), (1, 4), (16, 6)]
    meshes = [W.Mesh2D.uniform_rect(m, -1.0, 1.0, m, -1.0, 1.0) for m, _ in shapes]
    omegas = rng.uniform(2.0, 8.0, len(shapes))
    F = [rng.standard_normal(3 * m * m * n * n) / m for m, n in shapes]
    W0 = [rng.standard_normal(f.size) for f in F]
    warm = [0, 1, 0, 1, 1, 0, 1, 0]
    got = []
    for explicit in (False, True):
        systems = [W.WaveSystem(mesh, n, None, precision=precision) for mesh, (_, n) in zip(meshes, shapes)]
        systems[5].set_max_ctas(4)
        b = WaveHoltzBatch(systems, omegas)
        if explicit:
            b.set_launch(1, 2)
        runs = []
        for kw in (dict(maxit=3), dict(maxit=2, warm=warm), dict(maxit=2, warm=warm, pi0_norm=np.where(warm, 2.0, 0.0))):
            w, it, res, st = b.solve(F, tol=1e-12, W=[x.copy() for x in W0], **kw)
            runs.append((w, it.copy(), res.copy(), st.copy(), b.pi0_norm.copy()))
        got.append(runs)
    for (wa, ia, ra, sa, pa), (wb, ib, rb, sb, pb) in zip(*got):
        assert np.array_equal(ia, ib) and np.array_equal(sa, sb)
        assert np.allclose(ra, rb, rtol=1e-9, atol=0) and np.allclose(pa, pb, rtol=1e-12, atol=0)
        for x, y in zip(wa, wb):
            assert np.linalg.norm(x - y) <= 1e-12 * np.linalg.norm(y)


@pytest.mark.parametrize("n", [3, 5, 8])
def test_waveholtz_period(gpu_lib, n):
    import wavedg_b200 as W

    a, b, u, _ = _pair(9, 8, n, "fp64", 5)
    wa, wb = (W.WaveHoltz(9.0, s.mesh, n, None, approx_quad=True, system=s) for s in (a, b))
    for f in (lambda w, x: w.pi0(x, u), lambda w, x: w.S(x)):
        x, y = u.copy(), u.copy()
        f(wa, x)
        f(wb, y)
        # the forcing is added before the face terms here and after them there
        assert np.linalg.norm(x - y) <= 1e-13 * np.linalg.norm(y)
