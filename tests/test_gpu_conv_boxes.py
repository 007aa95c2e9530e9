"""The convolution kernels at the edges of their boxes (8 x 8 in (y, x), 2 to 8
planes), channel tiles and copy stages, against the same operation in 64 bits.
Bounds: a BF16 result is off by at most half a unit in its last place (2^-9
relative) plus the FP32 sum's error, at most k 2^-23 of the sum of the products'
magnitudes over its k terms; FP32 results have the latter alone."""
import ctypes as C

import pytest

import learned

pytestmark = pytest.mark.gpu


def _p(t):
    return C.c_void_p(t.data_ptr())


def _inputs(dims, cin, cout, seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    r = lambda *s: torch.randn(s, generator=g, device="cuda")
    return (r(*dims, cin).bfloat16(), (0.1 * r(cout, 27, cin)).bfloat16(), r(cout), r(*dims, cout).bfloat16())


def _shift(x, t):
    import torch
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    a, b, c = t // 9, t // 3 % 3, t % 3
    return p[:, a:a + x.shape[1], b:b + x.shape[2], c:c + x.shape[3]]


DIMS = [(1, 2, 8, 8), (2, 8, 8, 8), (1, 9, 7, 17), (3, 3, 3, 3), (1, 1, 8, 24), (2, 16, 24, 8), (1, 40, 16, 16)]


@pytest.mark.parametrize("cin,cout", [(16, 16), (48, 32), (64, 64), (128, 16), (16, 96)])
@pytest.mark.parametrize("dims", DIMS)
def test_conv_boxes(gpu, dims, cin, cout):
    import torch
    L = learned.klib()
    x, w, bias, _ = _inputs(dims, cin, cout, sum(dims) + cin)
    xd, wd = x.double(), w.double()
    ref = sum(_shift(xd, t) @ wd[:, t].T for t in range(27))
    mag = sum(_shift(xd.abs(), t) @ wd[:, t].abs().T for t in range(27))
    acc = (27 * cin + 4) * 2.0 ** -23
    for flags in (0, 1, 2, 4, 6):
        b = None if flags == 0 else bias
        f32 = bool(flags & 4)
        # a window at channel 16 of a wider buffer
        out = torch.full((*dims, cout + 32), 0.5, device="cuda", dtype=torch.float32 if f32 else torch.bfloat16)
        rc = L.xcnn_conv3d(_p(x), cin, 0, cin, _p(w), None if b is None else _p(b), _p(out), cout + 32, 16, cout, *dims,
                           flags, None)
        assert rc == 0
        torch.cuda.synchronize()
        y = ref if b is None else ref + b.double()
        if flags & 1:
            y = torch.relu(y)
        if flags & 2:
            y = y + 0.5
        tol = acc * (mag + (0 if b is None else b.double().abs()) + 0.5) + (0 if f32 else 2.0 ** -8 * y.abs())
        assert bool(((out[..., 16:16 + cout].double() - y).abs() <= tol).all()), (dims, flags)
        assert bool((out[..., :16] == 0.5).all()) and bool((out[..., 16 + cout:] == 0.5).all())


@pytest.mark.parametrize("cin,cout", [(16, 16), (32, 128), (48, 32), (16, 64)])
@pytest.mark.parametrize("dims", DIMS)
def test_weight_and_bias_gradients(gpu, dims, cin, cout):
    import torch
    L = learned.klib()
    x, _, _, g = _inputs(dims, cin, cout, 7 * sum(dims) + cin)
    nvox = g.numel() // cout
    flat = g.double().reshape(-1, cout)
    for odd in (0, 1):  # dw on an 8-byte boundary or between two
        buf = torch.zeros(cout * 27 * cin + 1, device="cuda")
        dw = buf[odd:odd + cout * 27 * cin]
        db = torch.zeros(cout, device="cuda")
        assert L.xcnn_conv3d_wgrad(_p(x), cin, 0, cin, _p(g), cout, 0, cout, _p(dw), *dims, None) == 0
        assert L.xcnn_bias_grad(_p(g), cout, 0, cout, nvox, _p(db), None) == 0
        torch.cuda.synchronize()
        dw = dw.double().reshape(cout, 27, cin)
        for t in range(27):
            xs = _shift(x.double(), t).reshape(-1, cin)
            tol = (nvox + 4) * 2.0 ** -23 * (flat.abs().T @ xs.abs())
            assert bool(((dw[:, t] - flat.T @ xs).abs() <= tol).all()), t
        assert bool(((db.double() - flat.sum(0)).abs() <= (nvox + 4) * 2.0 ** -23 * flat.abs().sum(0)).all())


@pytest.mark.parametrize("c,cs,c0", [(16, 16, 0), (32, 48, 16), (8, 24, 8), (4, 20, 12), (1, 3, 1)])
def test_relu_mask_and_bias_gradient_widths(gpu, c, cs, c0):
    """Widths that take 16-byte pieces and widths that do not."""
    import torch
    L = learned.klib()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(c)
    nvox = 1237
    g = torch.randn((nvox, cs), generator=gen, device="cuda").bfloat16()
    act = torch.randn((nvox, cs), generator=gen, device="cuda").bfloat16()
    want = g.clone()
    want[:, c0:c0 + c] = torch.where(act[:, c0:c0 + c] > 0, g[:, c0:c0 + c], torch.zeros_like(g[:, c0:c0 + c]))
    assert L.xcnn_relu_bwd(_p(g), cs, c0, _p(act), cs, c0, c, nvox, None) == 0
    db = torch.zeros(c, device="cuda")
    assert L.xcnn_bias_grad(_p(g), cs, c0, c, nvox, _p(db), None) == 0
    torch.cuda.synchronize()
    assert torch.equal(g, want)
    w = want[:, c0:c0 + c].double()
    assert bool(((db.double() - w.sum(0)).abs() <= (nvox + 4) * 2.0 ** -23 * w.abs().sum(0)).all())
