"""The transpose kernel, and convolutions computed on channels-last copies."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


# partial tiles on both sides, every vector width on either side, one row or column, misaligned storage
@pytest.mark.parametrize("batch,rows,cols", [(2, 64, 64), (3, 72, 784), (1, 8, 49), (2, 40, 196), (3, 256, 62), (2, 49, 72),
                                             (2, 196, 8), (1, 65, 64), (2, 130, 24), (1, 1, 8), (3, 7, 5), (1, 63, 129)])
@pytest.mark.parametrize("offset", [0, 1])
def test_transpose(batch, rows, cols, offset):
    from actnn_b200 import _lib
    x = torch.randint(-2 ** 15, 2 ** 15, (batch * rows * cols + offset,), dtype=torch.int16, device="cuda")[offset:]
    buf = torch.full((batch * rows * cols + 128,), 77, dtype=torch.int16, device="cuda")
    _lib.call("actnn_transpose16", x, x.data_ptr(), buf[64:].data_ptr(), batch, rows, cols, _lib.stream_of(x))
    ref = x.view(batch, rows, cols).transpose(1, 2).reshape(-1)
    assert torch.equal(buf[64:64 + ref.numel()], ref)
    assert (buf[:64] == 77).all() and (buf[64 + ref.numel():] == 77).all()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("c,k,h,ks,stride,pad,dil,bias", [(16, 24, 14, 3, 1, 1, 1, True), (8, 8, 7, 3, 2, 1, 1, False),
                                                          (64, 32, 9, (1, 3), 1, (0, 1), 1, False), (24, 40, 21, 5, 1, 2, 1, True),
                                                          (32, 32, 16, 3, 1, 2, 2, False)])
def test_convolution_against_64_bit(c, k, h, ks, stride, pad, dil, bias, dtype, monkeypatch):
    import actnn_b200 as actnn
    from actnn_b200.cpp_extension import backward_func as bf
    monkeypatch.setattr(bf, "CHANNELS_LAST_ELEMENTS", 0)          # small inputs keep NCHW otherwise
    from actnn_b200.conf import config
    torch.manual_seed(c + k)
    layer = actnn.QConv2d(c, k, ks, stride, pad, dil, bias=bias).cuda().to(dtype)
    x = torch.randn(6, c, h, h, device="cuda").to(dtype).requires_grad_()
    saved = dict(config.__dict__)
    try:
        config.compress_activation = False                        # exact saved input: only the convolution is compared
        y = layer(x)
        gy = torch.randn(y.shape, device="cuda").to(dtype)
        grads = torch.autograd.grad(y, [x] + list(layer.parameters()), gy)
    finally:
        config.__dict__.update(saved)
    assert y.is_contiguous() and all(g.is_contiguous() for g in grads)
    xd = x.detach().double().requires_grad_()
    params = [p.detach().double().requires_grad_() for p in layer.parameters()]
    yd = F.conv2d(xd, params[0], params[1] if bias else None, stride, pad, dil)
    ref = torch.autograd.grad(yd, [xd] + params, gy.double())
    eps = 2 ** -11 if dtype == torch.float16 else 2 ** -8
    for a, b in zip((y, *grads), (yd, *ref)):                      # float32 sums rounded once (the bias sum of a 16-bit tensor too)
        assert (a.double() - b).norm() <= 2 * eps * b.norm()
