"""The SMs that a batch's resident periods are given: never above a handle's CTA limit, together never
above the chip, and all of it where the solves have the groups."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _shares(shapes, precision="fp32"):
    import wavedg_b200 as W

    systems = []
    for m, n, cap in shapes:
        s = W.WaveSystem(W.Mesh2D.uniform_rect(m, -1.0, 1.0, m, -1.0, 1.0), n, None, precision=precision)
        if cap:
            s.set_max_ctas(cap)
        systems.append(s)
    b = W.WaveHoltzBatch(systems, np.full(len(shapes), 6.0))
    c = np.zeros(len(shapes), dtype=np.int32)
    assert W.lib().wdg_test_whbatch_shares(b._h, c.ctypes.data) == 0
    b.set_launch(1, 2)
    none = np.full(len(shapes), 7, dtype=np.int32)
    assert W.lib().wdg_test_whbatch_shares(b._h, none.ctypes.data) == 0
    assert not none.any()  # a chosen launch shape streams
    return c


@pytest.mark.parametrize("shapes", [[(40, 3, 4)], [(96, 4, 32), (12, 5, 0)], [(128, 4, 64)], [(9, 5, 1), (9, 5, 2), (40, 4, 3)],
                                    [(64, 4, 0), (96, 5, 0), (64, 7, 30), (128, 4, 70)]])
def test_shares(gpu_lib, shapes):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    c = _shares(shapes)
    assert 0 < c.sum() <= sms
    for got, (m, n, cap) in zip(c, shapes):
        assert 0 <= got <= (cap or sms)


def test_free_solves_fill_the_chip(gpu_lib):
    import torch

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert _shares([(64, 4, 0), (48, 5, 0)]).sum() == sms


def test_autotune_times_what_the_solves_run(gpu_lib):
    """Where every solve is resident the launch shape stays and the time is the resident steps', several times
    below the streaming launches'; a mixed batch tunes for the solve that streams."""
    import wavedg_b200 as W

    def batch(shapes):
        systems = [W.WaveSystem(W.Mesh2D.uniform_rect(m, -1.0, 1.0, m, -1.0, 1.0), n, None, precision="fp32")
                   for m, n in shapes]
        return systems, W.WaveHoltzBatch(systems, np.full(len(shapes), 9.0))

    _, a = batch([(32, 4), (24, 5)])
    before = a.launch_config()
    ms = a.autotune(64)
    assert a.launch_config() == before
    _, b = batch([(32, 4), (24, 5)])
    b.set_launch(1, 2)
    assert 0.0 < ms < 0.7 * b.autotune(64)
    _, c = batch([(330, 3), (20, 4)])  # the first is too large for the chip
    shares = np.zeros(2, dtype=np.int32)
    assert W.lib().wdg_test_whbatch_shares(c._h, shares.ctypes.data) == 0
    assert shares[0] == 0 and shares[1] > 0
    assert c.autotune(32) > 0.0
