"""Weight gradients of volumes whose planes lie more than 2^31 elements apart
over a box: 16 channels in a wide buffer.  Against the same operation in 64
bits; the FP32 sum's error is at most k 2^-23 of the sum of the products'
magnitudes over its k terms."""
import ctypes as C

import pytest

import learned

pytestmark = pytest.mark.gpu


def _p(t):
    return C.c_void_p(t.data_ptr())


def _shift(x, t):
    import torch
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    a, b, c = t // 9, t // 3 % 3, t % 3
    return p[:, a:a + x.shape[1], b:b + x.shape[2], c:c + x.shape[3]]


@pytest.mark.parametrize("dims", [(1, 2, 424, 424), (1, 3, 419, 423)])
@pytest.mark.parametrize("cout,wide_input", [(16, True), (128, True), (16, False)])
def test_weight_gradient_of_wide_planes(gpu, dims, cout, wide_input):
    import torch
    L = learned.klib()
    cin, wide, c0 = 16, 4096, 2032
    assert 3 * dims[2] * dims[3] * wide > 2 ** 31 - 1
    gen = torch.Generator(device="cuda")
    gen.manual_seed(cout)
    x, g = (torch.randn((*dims, c), generator=gen, device="cuda").bfloat16() for c in (cin, cout))
    big = torch.zeros((*dims, wide), dtype=torch.bfloat16, device="cuda")
    src = x if wide_input else g
    big[..., c0:c0 + src.shape[-1]] = src
    dw = torch.zeros((cout, 27, cin), device="cuda")
    torch.cuda.synchronize()
    a = (_p(big), wide, c0) if wide_input else (_p(x), cin, 0)
    b = (_p(g), cout, 0) if wide_input else (_p(big), wide, c0)
    assert L.xcnn_conv3d_wgrad(*a, cin, *b, cout, _p(dw), *dims, None) == 0
    torch.cuda.synchronize()
    flat = g.double().reshape(-1, cout)
    nvox = flat.shape[0]
    for t in range(27):
        xs = _shift(x.double(), t).reshape(-1, cin)
        tol = (nvox + 4) * 2.0 ** -23 * (flat.abs().T @ xs.abs())
        assert bool(((dw[:, t].double() - flat.T @ xs).abs() <= tol).all()), t
