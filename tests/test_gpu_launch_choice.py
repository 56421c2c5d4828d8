"""What a caller chose about a handle's launches, and its taking back: 0 elements per block, 0 stages and
kernel -1 each mean the built-in default, with which a mesh that fits the chip stays on it."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def _ctas(s, forced=0):
    import wavedg_b200 as W

    n = C.c_int(-1)
    assert W.lib().wdg_test_resident(s._h, forced, C.byref(n)) == 0
    return n.value


def test_defaults_are_not_choices(gpu_lib):
    import wavedg_b200 as W

    s = W.WaveSystem(W.Mesh2D.uniform_rect(24, -1.0, 1.0, 20, -1.0, 1.0), 5, None)
    chunk = s.tile
    default = _ctas(s)
    assert default > 0
    s.tile = 0
    s.set_stages(0)
    assert _ctas(s) == default
    s.tile = 2 * chunk
    assert _ctas(s) == 0
    s.set_stages(3)
    s.tile = 0
    assert s.tile == chunk and _ctas(s) == 0  # the depth is still the caller's
    s.set_stages(0)
    assert _ctas(s) == default
    s.set_kernel(2)
    s.tile = 0
    s.set_stages(0)
    assert _ctas(s) == 0  # and so is the kernel
    s.set_kernel(-1)
    assert _ctas(s) == default
    with pytest.raises(W.WdgError):
        s.tile = 7
    assert _ctas(s) == default
    s.set_max_ctas(9)
    assert 0 < _ctas(s) <= 9


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_state_steps_need_a_state(gpu_lib, precision):
    import numpy as np

    import wavedg_b200 as W

    s = W.WaveSystem(W.Mesh2D.uniform_rect(6, -1.0, 1.0, 5, -1.0, 1.0), 4, None, precision=precision)
    assert s.step_state(1e-3, 0.5, 0) == 0.5
    with pytest.raises(W.WdgError) as e:
        s.step_state(1e-3, 0.0, 1)
    assert e.value.code == W._lib.WDG_ERR_ARG
    s.upload(np.ones(s.ndof))
    s.step_state(1e-3, 0.0, 1)
    assert np.isfinite(s.download()).all()


def test_step_kernel(gpu_lib):
    import wavedg_b200 as W

    small, large = (W.WaveSystem(W.Mesh2D.uniform_rect(k, -1.0, 1.0, k, -1.0, 1.0), 5, None) for k in (20, 180))
    assert (small.step_kernel(), large.step_kernel()) == ("resident", "line")
    for s in (small, large):
        s.set_kernel(2)
        assert s.step_kernel() == "ws"
        s.set_kernel(1)
        assert s.step_kernel() == "tiled"
        s.set_kernel(0)
        assert s.step_kernel() == "warp"
        s.set_kernel(-1)
    large.set_max_ctas(40)
    assert large.step_kernel() == "ws"
