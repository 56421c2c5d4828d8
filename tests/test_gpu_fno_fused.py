"""The Fourier layer's fused launches against the same network with its GEMMs and elementwise passes apart:
the forward pass and the gradients at every layer bit for bit (the same products in the same order), the
weight gradients, whose split sums meet in atomics, to FP32 rounding.  Grids that end inside a tile, widths
below the tile, and a network the fused tile does not take."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G,width,modes,H,B", [(24, 8, 4, 16, 1), (136, 24, 12, 40, 2), (160, 32, 16, 64, 1), (48, 16, 8, 8, 3)])
def test_fused_matches_separate(gpu_lib, G, width, modes, H, B):
    import torch

    from wavedg_b200 import fno

    rng = np.random.default_rng(G)
    inp = torch.from_numpy(rng.standard_normal((B, 4, G, G))).to("cuda", torch.float32)
    dy = torch.from_numpy(rng.standard_normal((B, 3, G, G))).to("cuda", torch.float32)
    out = []
    for fused in (True, False):
        net = fno.FNO(grid=G, width=width, modes=modes, layers=3, hidden=H, seed=2)
        assert net._fused()
        if not fused:
            net._fused = lambda: False
        assert torch.equal(net.forward(inp), net.forward(inp, keep=True))
        y = net.forward(inp, keep=True)
        net.backward(dy)
        out.append((y.clone(), {k: g.clone() for k, g in net.grads.items()}))
    (ya, ga), (yb, gb) = out
    assert torch.equal(ya, yb)
    for k in ga:
        if k[0] == "b" or k[0] == "R" or k.endswith("_b"):
            assert torch.equal(ga[k], gb[k]), k
        else:  # sums of at most 3 * 160^2 products in FP32, in another order each time
            assert float((ga[k] - gb[k]).norm() / gb[k].norm()) < 1e-5, k


def test_wide_network_takes_the_separate_path(gpu_lib):
    import torch

    from wavedg_b200 import fno

    net = fno.FNO(grid=40, width=40, modes=18, layers=2, hidden=16, seed=2)
    assert not net._fused()
    x = torch.randn(1, 4, 40, 40, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    y = net.forward(x, keep=True)
    net.backward(torch.ones_like(y))
    assert torch.isfinite(y).all() and all(torch.isfinite(g).all() for g in net.grads.values())
