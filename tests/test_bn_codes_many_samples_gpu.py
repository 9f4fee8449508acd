"""Batch norm on the codes where a warp walks many samples: from one to the next, past a block of 32, and the octets
requested ahead in the forward pass of large 16-bit activations."""
import pytest
import torch

from test_bn_codes_gpu import EPS, backward64, compressed

pytestmark = pytest.mark.gpu

F16, BF16, F32 = torch.float16, torch.bfloat16, torch.float32
# 40 samples and more a warp: whole groups, and a last group that is not whole.  Seven and more, and 2^24 elements: whole
# groups, samples that end in a part of a group, channels that change inside octets, octets on 8 bytes (none ahead)
CASES = [((2000, 64, 784), F16), ((2000, 60, 784), BF16), ((2000, 64, 784), F32), ((2000, 60, 784), F32),
         ((400, 64, 784), F16), ((400, 60, 784), F16), ((400, 40, 1225), BF16), ((200, 100, 1225), F16)]
CHAIN = 4 * 64 + 64              # float32 additions in a row: four a sample and octet over the samples of a warp, then trees


@pytest.mark.parametrize("shape,dtype", CASES)
def test_backward(shape, dtype):
    from actnn_b200.cpp_extension import backward_func as bf
    n, c, hw = shape
    x, quantized, x_hat = compressed(n, c, hw, dtype)
    dy = torch.randn(n, c, hw, device="cuda").to(dtype)
    weight = torch.rand(c, device="cuda") + 0.5
    mean = x.float().mean((0, 2))
    invstd = 1 / torch.sqrt(x.float().var((0, 2), unbiased=False) + 1e-5)
    dx, dw, db = bf.batch_norm_codes_backward(quantized, shape, dtype, dy, weight, mean, invstd)
    rx, rw, rb = backward64(x_hat, dy, weight, mean, invstd)
    away = (x_hat.double() - mean.double().view(1, -1, 1)).abs()
    assert ((db.double() - rb).abs() <= CHAIN * 2 ** -24 * dy.double().abs().sum((0, 2))).all()
    assert ((dw.double() - rw).abs() <= CHAIN * 2 ** -24 * (dy.double().abs() * away).sum((0, 2)) * invstd.double()).all()
    # a few float32 operations on values of order |w i| * max|dy|, then one rounding to the type
    scale = (weight * invstd).double().view(1, -1, 1)
    big = scale * (dy.double().abs().max() + away * invstd.double().view(1, -1, 1))
    assert ((dx.double() - rx).abs() <= (EPS[dtype] * 1.01 + CHAIN * 2 ** -24) * big + 1e-7).all()


@pytest.mark.parametrize("shape,dtype", CASES)
def test_forward(shape, dtype):
    from actnn_b200.cpp_extension import backward_func as bf
    from actnn_b200.cpp_extension import quantization as q
    n, c, hw = shape
    torch.manual_seed(1)
    x = (torch.randn(n, c, hw, device="cuda") * 1.5 + torch.linspace(-8, 8, c, device="cuda").view(1, c, 1)).to(dtype)
    weight, bias = torch.rand(c, device="cuda") + 0.5, torch.randn(c, device="cuda")
    gen = torch.cuda.default_generators[torch.cuda.current_device()]
    gen.manual_seed(9)
    gen.set_offset(4)
    y, quantized, mean, invstd = bf.batch_norm_codes_forward(x, weight, bias, None, None, 0.1, 1e-5, 2 * n, 8, 0.5, True)
    stat = BF16 if dtype == F32 else dtype
    f, kw = c * hw, dict(philox=(9, 4), stat_dtype=stat)
    if f % 256:
        ref = q.compress_mixed_samples(x.view(n, f), 2 * n, 8, 0.5, **kw)
    else:
        ref = q.compress_mixed_precision(x.view(n, f // 256, 256), 2 * n, 8, 0.5, **kw)
    assert all(torch.equal(a, b) for a, b in zip(quantized, ref))          # the codec to the bit
    assert torch.equal(y, bf.batch_norm_elemt(x, weight, bias, mean, invstd, 1e-5))
    m, v = x.double().mean((0, 2)), x.double().var((0, 2), unbiased=False)
    # float32 sums of |x - shift| and its square, the shift within five deviations of the mean
    assert ((mean.double() - m).abs() <= CHAIN * 2 ** -24 * (6 * torch.sqrt(v) + m.abs())).all()
    assert ((invstd.double() * torch.sqrt(v + 1e-5) - 1).abs() <= CHAIN * 2 ** -24 * 48).all()
