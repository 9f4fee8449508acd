"""Pooling gradients of 16-bit types to the bit: terms in the order of the windows from +0 in float32, one rounding."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def reference(gy, idx, shape, k, p):
    n, c, h, w = shape
    ho_n, wo_n = gy.shape[2:]
    acc = torch.zeros(shape, dtype=torch.float32)
    rows, cols = torch.arange(h).view(h, 1), torch.arange(w).view(1, w)
    for a in range(2):
        ho = torch.div(rows + p - k + 2, 2, rounding_mode="floor") + a           # ceil((row + p - k + 1) / 2), then the next
        for b in range(2):
            wo = torch.div(cols + p - k + 2, 2, rounding_mode="floor") + b
            kh, kw = rows + p - 2 * ho, cols + p - 2 * wo
            ok = (ho >= 0) & (ho < ho_n) & (wo >= 0) & (wo < wo_n) & (kh >= 0) & (kh < k) & (kw >= 0) & (kw < k)
            at = (ho.clamp(0, ho_n - 1) * wo_n + wo.clamp(0, wo_n - 1)).view(1, 1, -1).expand(n, c, -1)
            g = gy.view(n, c, -1).gather(2, at).view(shape).float()
            code = idx.view(n, c, -1).gather(2, at).view(shape).int()
            acc = torch.where(ok & (code == kh * k + kw), acc + g, acc)
    return acc.to(gy.dtype)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("h,w", [(1, 8), (7, 16), (16, 24), (33, 40), (112, 16)])
@pytest.mark.parametrize("k,p", [(2, 0), (2, 1), (3, 0), (3, 1)])
@pytest.mark.parametrize("offset", [0, 1])
def test_gradient_to_the_bit(k, p, h, w, dtype, offset):
    from actnn_b200.cpp_extension import quantization as q
    if h + 2 * p < k:
        pytest.skip("no output")
    torch.manual_seed(h * w + k)
    x = torch.randint(-2, 3, (3, 4, h, w)).to(dtype)                             # ties: windows share their maxima
    geom = ((k, k), (2, 2), (p, p), (1, 1))
    y, idx = q.max_pool2d_forward(x.cuda(), *geom)
    gy = torch.randn(y.shape) * 2.0 ** torch.randint(-26, 15, y.shape).float()    # subnormals to overflow
    special = torch.tensor([-0.0, 0.0, float("inf"), float("-inf"), float("nan"), 1e-7])
    gy = torch.where(torch.rand(y.shape) < 0.2, special[torch.randint(6, y.shape)], gy).to(dtype)
    base = torch.empty(gy.numel() + offset, dtype=dtype, device="cuda")
    base[offset:] = gy.view(-1).cuda()
    gx = q.max_pool2d_backward(base[offset:].view(gy.shape), idx, x.shape, *geom).cpu()
    want = reference(gy, idx.cpu(), x.shape, k, p)
    nan = torch.isnan(want)
    assert torch.equal(torch.isnan(gx), nan)
    assert torch.equal(gx.view(torch.int16)[~nan], want.view(torch.int16)[~nan])
