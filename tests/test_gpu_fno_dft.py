"""The truncated DFT along y on every route of its kernels: pairs read and written whole or, off an 8-byte
boundary, value by value; rows and twiddles in shared memory or too long for it; more blocks than
a grid has along y.  Against the same sums in complex FP64.

Tolerance 1e-5 (relative 2-norm): FP32 twiddles and at most 12400 ordered FP32 sums of random values,
whose roundings (6e-8 each) add up like a random walk."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _call(x, G, K, KX, inverse, sign, shift, bf16=False):
    import torch

    import wavedg_b200 as W

    B = x.shape[0]
    m = torch.arange(G, dtype=torch.float64)
    cs, sn = (f(2 * np.pi * m / G).to("cuda", torch.float32) for f in (torch.cos, torch.sin))
    src = torch.zeros(x.numel() * 2 + shift, dtype=torch.float32, device="cuda")[shift:]
    src.copy_(torch.view_as_real(x).reshape(-1))
    rows = G if inverse else K
    out = torch.zeros(B * rows * KX * 2 + shift, dtype=torch.float32, device="cuda")[shift:]
    outb = torch.zeros(B * rows * KX * 2 + shift, dtype=torch.bfloat16, device="cuda")[shift:]
    p = lambda t: C.c_void_p(t.data_ptr())
    st = W.lib().wdg_fno_dft_y(p(src), p(out), p(outb) if bf16 else None, p(cs), p(sn), B, G, K, KX, inverse, float(sign),
                               C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0, W.lib().wdg_last_error()
    torch.cuda.synchronize()
    re, im = out.reshape(B, rows, KX, 2).unbind(-1)
    return torch.complex(re, im), outb.float(), out


def _twiddles(G, K, sign):
    import torch

    k = torch.arange(K, dtype=torch.float64)
    ky = torch.where(k < K // 2, k, k - K)
    y = torch.arange(G, dtype=torch.float64)
    ph = (ky[:, None] * y[None]) % G
    return torch.polar(torch.ones(K, G, dtype=torch.float64), sign * 2 * np.pi * ph / G).cuda()


# (B, G, K, KX): the usual; odd sizes; a row longer than shared memory; a table longer than it
@pytest.mark.parametrize("B,G,K,KX", [(3, 24, 8, 4), (2, 37, 6, 5), (1, 6, 2, 12300), (1, 12400, 2, 3), (2, 5, 8, 3)])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("inverse", [0, 1])
def test_against_fp64(gpu_lib, B, G, K, KX, shift, inverse):
    import torch

    g = torch.Generator("cuda").manual_seed(G)
    x = torch.randn(B, K if inverse else G, KX, dtype=torch.complex64, device="cuda", generator=g)
    sign = 1.0 if inverse else -1.0
    T = _twiddles(G, K, sign)
    ref = torch.einsum("ky,bkx->byx" if inverse else "ky,byx->bkx", T, x.to(torch.complex128))
    got, outb, out = _call(x, G, K, KX, inverse, sign, shift, bf16=bool(inverse))
    assert float((got - ref).abs().norm() / ref.abs().norm()) < 1e-5
    if inverse:
        assert torch.equal(outb, out.to(torch.bfloat16).float())


@pytest.mark.parametrize("G,KX,inverse", [(2, 8388608 + 300, 0), (2097152 + 65, 1, 1)])
def test_more_blocks_than_a_grid_has(gpu_lib, G, KX, inverse):
    import torch

    g = torch.Generator("cuda").manual_seed(1)
    x = torch.randn(1, 2, KX, dtype=torch.complex64, device="cuda", generator=g)
    sign = 1.0 if inverse else -1.0
    ref = torch.einsum("ky,bkx->byx" if inverse else "ky,byx->bkx", _twiddles(G, 2, sign), x.to(torch.complex128))
    got, _, _ = _call(x, G, 2, KX, inverse, sign, 0)
    assert float((got - ref).abs().norm() / ref.abs().norm()) < 1e-5
