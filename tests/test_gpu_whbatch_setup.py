"""A batch whose set-up of the resident periods fails part of the way (a host-made allocation error,
nothing else goes wrong) reports it, and the next solve completes the set-up and is right."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(precision="fp64"):
    import wavedg_b200 as W

    meshes = [W.Mesh2D.uniform_rect(m, -1.0, 1.0, m, -1.0, 1.0) for m in (12, 7)]
    systems = [W.WaveSystem(mesh, n, None, precision=precision) for mesh, n in zip(meshes, (5, 4))]
    rng = np.random.default_rng(3)
    return W.WaveHoltzBatch(systems, [6.0, 5.0]), [rng.standard_normal(s.ndof) for s in systems]


# the set-up makes one record, then five parts per solve
@pytest.mark.parametrize("call", [1, 2, 3, 4, 5, 6, 7, 11])
def test_solve_after_a_failed_set_up(gpu_lib, call):
    import wavedg_b200 as W

    b, F = _batch()
    want = b.solve(F, tol=1e-12, maxit=2)[0]
    b, F = _batch()
    assert W.lib().wdg_test_whbatch_fail(b._h, call) == 0
    with pytest.raises(W.WdgError):
        b.solve(F, tol=1e-12, maxit=2)
    got = b.solve(F, tol=1e-12, maxit=2)[0]
    for x, y in zip(got, want):
        assert np.array_equal(x, y)
    assert W.lib().wdg_test_whbatch_fail(b._h, -1) == W._lib.WDG_ERR_ARG
