"""Batch-norm passes that work on the compressed activation, against decode + 64-bit arithmetic."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# (N, C, HW): one channel per octet, per half octet, changes inside octets; a channel over several columns and many
# channels in a column; samples that are not whole groups; one sample; more samples than a block of 32
SHAPES = [(2, 64, 3136), (70, 24, 784), (5, 3, 40), (37, 32, 196), (3, 20, 12), (40, 7, 49), (33, 5, 225), (1, 130, 9),
          (6, 33, 8), (9, 2, 1600), (4, 3, 1029)]
EPS = {torch.float16: 2 ** -11, torch.bfloat16: 2 ** -8, torch.float32: 2 ** -24}


def compressed(n, c, hw, dtype, seed=0):
    from actnn_b200.cpp_extension import quantization as q
    torch.manual_seed(seed)
    x = (torch.randn(n, c, hw, device="cuda") * 1.5 + torch.linspace(-1, 1, c, device="cuda").view(1, c, 1)).to(dtype)
    stat = torch.bfloat16 if dtype == torch.float32 else dtype
    f = c * hw
    if f % 256:
        out = q.compress_mixed_samples(x.view(n, f), 2 * n, 8, 0.5, philox=(1, 4), stat_dtype=stat)
        x_hat = q.unpack_mixed_samples(out[0], out[1], out[2], out[3], (n, c, hw), out_dtype=dtype)
    else:
        out = q.compress_mixed_precision(x.view(n, f // 256, 256), 2 * n, 8, 0.5, philox=(1, 4), stat_dtype=stat)
        x_hat = q.unpack_mixed_precision(*out[:4], n, f // 256, 256, out_dtype=dtype).view(n, c, hw)
    return x, out[:4], x_hat


def backward64(x_hat, dy, weight, mean, invstd):
    x, g = x_hat.double(), dy.double()
    m, i, w = (t.double().view(1, -1, 1) for t in (mean, invstd, weight))
    cnt = x.shape[0] * x.shape[2]
    sdy, sdyx = g.sum((0, 2)), (g * (x - m)).sum((0, 2))
    dx = w * i * (g - sdy.view(1, -1, 1) / cnt - (x - m) * i * i * sdyx.view(1, -1, 1) / cnt)
    return dx, sdyx * i.view(-1), sdy


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("offset", [0, 1])
def test_backward_from_codes(shape, dtype, offset):
    from actnn_b200.cpp_extension import backward_func as bf
    n, c, hw = shape
    x, quantized, x_hat = compressed(n, c, hw, dtype)
    base = torch.randn(n * c * hw + offset, device="cuda").to(dtype)
    dy = base[offset:].view(n, c, hw)
    weight = torch.rand(c, device="cuda") + 0.5
    mean = x.float().mean((0, 2))
    invstd = 1 / torch.sqrt(x.float().var((0, 2), unbiased=False) + 1e-5)
    dx, dw, db = bf.batch_norm_codes_backward(quantized, shape, dtype, dy, weight, mean, invstd)
    rx, rw, rb = backward64(x_hat, dy, weight, mean, invstd)
    # sums of N * HW float32 terms of order one in chains and trees: well under 64 roundings of the sum of magnitudes
    mags = (dy.double().abs()).sum((0, 2)), (dy.double() * (x_hat.double() - mean.double().view(1, -1, 1))).abs().sum((0, 2))
    assert ((db.double() - rb).abs() <= 64 * 2 ** -24 * mags[0] + 1e-6).all()
    assert ((dw.double() - rw).abs() <= 64 * 2 ** -24 * mags[1] * invstd.double() + 1e-6).all()
    # dx: a few float32 operations on values of order |w i| * max|dy|, then one rounding to the type
    big = (weight * invstd).double().view(1, -1, 1) * (dy.double().abs().max() + (x_hat.double() - mean.double().view(1, -1, 1)).abs() * invstd.double().view(1, -1, 1))
    assert ((dx.double() - rx).abs() <= (EPS[dtype] * 1.01 + 64 * 2 ** -24) * big + 1e-7).all()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shape", SHAPES + [(1030, 8, 16)])
@pytest.mark.parametrize("stochastic", [True, False])
def test_forward(shape, dtype, stochastic):
    from actnn_b200.cpp_extension import backward_func as bf
    from actnn_b200.cpp_extension import quantization as q
    n, c, hw = shape
    torch.manual_seed(1)
    x = (torch.randn(n, c, hw, device="cuda") * 1.5 + torch.linspace(-8, 8, c, device="cuda").view(1, c, 1)).to(dtype)
    weight, bias = torch.rand(c, device="cuda") + 0.5, torch.randn(c, device="cuda")
    rm, rv = torch.randn(c, device="cuda"), torch.rand(c, device="cuda")
    rm0, rv0 = rm.double(), rv.double()
    gen = torch.cuda.default_generators[torch.cuda.current_device()]
    gen.manual_seed(9)
    gen.set_offset(4)
    y, quantized, mean, invstd = bf.batch_norm_codes_forward(x, weight, bias, rm, rv, 0.1, 1e-5, 2 * n, 8, 0.5, stochastic)
    f = c * hw
    stat = torch.bfloat16 if dtype == torch.float32 else dtype
    kw = dict(philox=(9, 4), stat_dtype=stat) if stochastic else dict(stochastic=False, stat_dtype=stat)
    if f % 256:
        ref = q.compress_mixed_samples(x.view(n, f), 2 * n, 8, 0.5, **kw)
    else:
        ref = q.compress_mixed_precision(x.view(n, f // 256, 256), 2 * n, 8, 0.5, **kw)
    assert all(torch.equal(a, b) for a, b in zip(quantized, ref))          # the codec to the bit
    xd = x.double()
    m, v = xd.mean((0, 2)), xd.var((0, 2), unbiased=False)
    i = 1 / torch.sqrt(v + 1e-5)
    # shifted float32 sums: 64 roundings of sums of |x - shift| and its square, shift within 4 deviations of the mean
    dev = torch.sqrt(v) + 1e-3
    assert ((mean.double() - m).abs() <= 64 * 2 ** -24 * (5 * dev + m.abs())).all()
    assert ((invstd.double() / i - 1).abs() <= 64 * 2 ** -24 * 25).all()
    cnt = n * hw
    assert torch.allclose(rm.double(), 0.9 * rm0 + 0.1 * m, rtol=1e-5, atol=1e-5)
    assert torch.allclose(rv.double(), 0.9 * rv0 + 0.1 * v * (cnt / (cnt - 1)), rtol=1e-4, atol=1e-6)
    ry = (xd - m.view(1, -1, 1)) * (i * weight.double()).view(1, -1, 1) + bias.double().view(1, -1, 1)
    big = ry.abs() + (xd - m.view(1, -1, 1)).abs() * (i * weight.double()).view(1, -1, 1) + bias.double().abs().view(1, -1, 1) \
        + (m.abs() * i * weight.double()).view(1, -1, 1)
    assert ((y.double() - ry).abs() <= (EPS[dtype] * 1.01 + 2048 * 2 ** -24) * big).all()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shape", [(2, 64, 3136), (9, 16, 800), (33, 3, 256), (70, 8, 288)])
def test_forward_from_statistics_of_a_pass_before_it(shape, dtype):
    """What maps of 256 and more whole groups take: ranges and statistics come from ``batch_norm_stats_minimax``."""
    from actnn_b200.cpp_extension import backward_func as bf
    from actnn_b200.cpp_extension import quantization as q
    n, c, hw = shape
    torch.manual_seed(2)
    x = (torch.randn(n, c, hw, device="cuda") * 1.5 + torch.linspace(-8, 8, c, device="cuda").view(1, c, 1)).to(dtype)
    weight, bias = torch.rand(c, device="cuda") + 0.5, torch.randn(c, device="cuda")
    rm, rv = torch.randn(c, device="cuda"), torch.rand(c, device="cuda")
    stats = bf.batch_norm_stats_minimax(x, weight, bias, rm, rv, 0.1, 1e-5)
    after = rm.clone(), rv.clone()
    gen = torch.cuda.default_generators[torch.cuda.current_device()]
    gen.manual_seed(9)
    gen.set_offset(4)
    y, quantized, mean, invstd = bf.batch_norm_codes_forward(x, weight, bias, rm, rv, 0.1, 1e-5, 2 * n, 8, 0.5, True, stats)
    assert torch.equal(rm, after[0]) and torch.equal(rv, after[1])          # updated once, by the pass before
    assert torch.equal(mean, stats[2]) and torch.equal(invstd, stats[3])
    stat = torch.bfloat16 if dtype == torch.float32 else dtype
    ref = q.compress_mixed_precision(x.view(n, c * hw // 256, 256), 2 * n, 8, 0.5, philox=(9, 4), stat_dtype=stat)
    assert all(torch.equal(a, b) for a, b in zip(quantized, ref))          # the codec to the bit
    assert torch.equal(y, bf.batch_norm_elemt(x, weight, bias, mean, invstd, 1e-5))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,c,h,w", [(20, 48, 14, 14), (6, 5, 9, 7), (40, 16, 16, 16), (12, 24, 2, 2), (3, 8, 1, 8)])
@pytest.mark.parametrize("affine", ["float32", "as the input"])
def test_layer_backward_takes_the_codes_and_agrees_with_the_decoded_path(monkeypatch, n, c, h, w, dtype, affine):
    """Maps of at least 8 positions take the codes, smaller ones the decoded path in both arms."""
    import actnn_b200 as actnn
    from actnn_b200.cpp_extension import backward_func as bf
    layer = actnn.QBatchNorm2d(c).cuda()
    if affine != "float32":
        layer.weight.data, layer.bias.data = layer.weight.data.to(dtype), layer.bias.data.to(dtype)
    x = torch.randn(n, c, h, w, device="cuda", dtype=dtype).requires_grad_()
    gy = torch.randn_like(x)
    real, results, taken = bf.batch_norm_codes_backward, [], []
    for use in (True, False):
        monkeypatch.setattr(bf, "batch_norm_codes_backward",
                            (lambda *a: (taken.append(real(*a)), taken[-1])[1]) if use else lambda *a: None)
        torch.manual_seed(5)
        results.append(torch.autograd.grad(layer(x), [x, layer.weight, layer.bias], gy))
    assert (taken[0] is not None) == (h * w >= 8)
    # sums in another order: 64 float32 roundings of sums of n * h * w terms of order one; then one rounding to the
    # type of the result, and of x's gradient another where its two sums' roundings moved it
    for a, b in zip(*results):
        assert a.dtype == b.dtype
        big = b.double().abs().max().item()
        bound = 2 * EPS[a.dtype] * b.double().abs() + 64 * 2 ** -24 * (big + (n * h * w) ** 0.5 * 4)
        assert ((a.double() - b.double()).abs() <= bound).all()


@pytest.mark.parametrize("hw", [14, 2])                       # from the codes; fewer than 8 positions: decoded
@pytest.mark.parametrize("frozen", [False, True])
def test_layer_without_trainable_weight_and_bias(hw, frozen):
    """``affine=False``, and affine parameters that need no gradient: only the input has one, that of weight 1 and
    bias 0."""
    import actnn_b200 as actnn
    x = torch.randn(12, 40, hw, hw, device="cuda", dtype=torch.float16).requires_grad_()
    gy = torch.randn_like(x)
    grads = []
    for trainable in (True, False):
        layer = actnn.QBatchNorm2d(40, affine=trainable or frozen).cuda()
        if not trainable:
            layer.requires_grad_(False)
        torch.manual_seed(5)
        x.grad = None
        layer(x).backward(gy)
        assert all((p.grad is not None) == trainable for p in layer.parameters())
        grads.append(x.grad)
    assert torch.equal(*grads)
