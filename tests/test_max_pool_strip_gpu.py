"""The strip kernels of 2x2 / 3x3 pooling at stride 2: edges of strips, segments and planes, ties, infinities and NaN."""
import pytest
import torch

import actnn_oracle as O

pytestmark = pytest.mark.gpu


# rows of one, two and five segments, the extra window of 2x2 with padding, odd heights, heights around a strip of eight
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("h,w", [(1, 8), (2, 16), (7, 24), (16, 8), (33, 40), (112, 16)])
@pytest.mark.parametrize("k,p", [(2, 0), (2, 1), (3, 0), (3, 1)])
def test_strips(k, p, h, w, dtype):
    from actnn_b200.cpp_extension import quantization as q
    if h + 2 * p < k:
        pytest.skip("no output")
    torch.manual_seed(h * w + k)
    x = torch.randint(-3, 4, (2, 3, h, w)).to(dtype)                       # many ties
    x[0, 1] = torch.randn(h, w).to(dtype)
    x[1, 0] = float("-inf")
    x[1, 1, :, ::3] = float("nan")
    x[1, 2] = -0.0
    x[1, 2, :, 1::2] = 0.0
    geom = ((k, k), (2, 2), (p, p), (1, 1))
    y, idx = q.max_pool2d_forward(x.cuda(), *geom)
    ry, ridx = O.max_pool2d_forward(x, *geom)
    assert torch.equal(y.cpu(), ry) and torch.equal(idx.cpu(), ridx)
    # a window without a finite value keeps code 0, which may name a tap in the padding: not for the oracle's scatter
    x[1] = torch.randn(3, h, w).to(dtype)
    idx, ridx = q.max_pool2d_forward(x.cuda(), *geom)[1], O.max_pool2d_forward(x, *geom)[1]
    gy = torch.randn(y.shape).to(dtype)
    gx = q.max_pool2d_backward(gy.cuda(), idx, x.shape, *geom)
    rgx = O.max_pool2d_backward(gy, ridx, x.shape, *geom)
    # at most four float32 terms in the oracle's order, rounded once: one unit in the last place
    eps = {torch.float16: 2 ** -10, torch.bfloat16: 2 ** -7, torch.float32: 2 ** -22}[dtype]
    assert ((gx.cpu().float() - rgx.float()).abs() <= eps * rgx.float().abs() + 1e-7).all()


@pytest.mark.parametrize("offset", [0, 1])
def test_many_planes_and_unaligned_gradient(offset):
    """Strips of the full length, and a gradient without vector alignment."""
    from actnn_b200.cpp_extension import quantization as q
    x = torch.randn(64, 96, 56, 56, dtype=torch.float16)
    geom = ((3, 3), (2, 2), (1, 1), (1, 1))
    y, idx = q.max_pool2d_forward(x.cuda(), *geom)
    ry, ri = torch.nn.functional.max_pool2d(x.cuda().float(), 3, 2, 1, return_indices=True)
    assert torch.equal(y.float(), ry)
    gy = torch.randn(y.numel() + offset, device="cuda").half()[offset:].view(y.shape)
    gx = q.max_pool2d_backward(gy, idx, x.shape, *geom)
    ref = torch.zeros(64 * 96, 56 * 56, device="cuda", dtype=torch.float64)
    ref.scatter_add_(1, ri.view(64 * 96, -1), gy.double().view(64 * 96, -1))
    assert ((gx.double().view_as(ref) - ref).abs() <= 2 ** -10 * ref.abs() + 1e-6).all()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("h,w", [(9, 16), (12, 24)])
@pytest.mark.parametrize("k,p", [(2, 0), (2, 1), (3, 0), (3, 1)])
def test_value_is_the_first_maximum_to_the_bit(k, p, h, w, dtype):
    """Windows whose maximum is a zero: the sign of the first zero, not that of a later one."""
    from actnn_b200.cpp_extension import quantization as q
    torch.manual_seed(h + k)
    x = torch.tensor([-0.0, 0.0, -1.0])[torch.randint(3, (3, 5, h, w))].to(dtype)
    geom = ((k, k), (2, 2), (p, p), (1, 1))
    y, idx = q.max_pool2d_forward(x.cuda(), *geom)
    ry, ridx = O.max_pool2d_forward(x, *geom)
    bits = torch.int32 if dtype == torch.float32 else torch.int16
    assert torch.equal(y.cpu().view(bits), ry.view(bits)) and torch.equal(idx.cpu(), ridx)
