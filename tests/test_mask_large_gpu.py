"""ReLU and dropout on tensors from the size on at which every warp takes one block of 1024 elements."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# input and output together just over 160 MiB; the last block whole, of 256 elements, and of 77
SIZES = [(torch.float16, 41 << 20), (torch.bfloat16, (40 << 20) + 1024 + 256), (torch.float16, (40 << 20) + 1024 + 77),
         (torch.float32, (20 << 20) + 1024 + 256), (torch.float32, (20 << 20) + 1024 + 77)]


def bitmask(keep):
    """Bit k of byte e // 8 is element 8 * (e // 8) + k, padded with zero bits to whole words."""
    bits = torch.zeros(-(-keep.numel() // 32) * 32, dtype=torch.uint8, device=keep.device)
    bits[:keep.numel()] = keep
    weights = torch.tensor([1, 2, 4, 8, 16, 32, 64, 128], dtype=torch.uint8, device=keep.device)
    return (bits.view(-1, 8) * weights).sum(1, dtype=torch.uint8).view(torch.int32)


@pytest.mark.parametrize("dtype,numel", SIZES)
def test_relu(dtype, numel):
    from actnn_b200.cpp_extension import quantization as q
    torch.manual_seed(numel % 1000)
    x, dy = (torch.randn(numel, device="cuda", dtype=dtype) for _ in range(2))
    want, keep = torch.relu(x), x > 0
    y, mask = q.relu_forward(x)
    assert torch.equal(y, want) and torch.equal(mask, bitmask(keep))
    assert torch.equal(q.relu_backward(dy, mask), torch.where(keep, dy, torch.zeros_like(dy)))
    if numel % 256 == 0:
        y, again, mn, mx = q.relu_forward(x, with_minmax=True)
        assert torch.equal(y, want) and torch.equal(again, mask)
        assert torch.equal(mn, want.view(-1, 256).amin(1)) and torch.equal(mx, want.view(-1, 256).amax(1))


@pytest.mark.parametrize("dtype,numel", SIZES)
def test_dropout(dtype, numel):
    from actnn_b200.cpp_extension import quantization as q
    torch.manual_seed(numel % 1000)
    x, p = torch.randn(numel, device="cuda", dtype=dtype), 0.5              # 1 / (1 - p) is exact
    keep = q.dropout_uniform_fill(numel, "cuda", 31, 8) > p
    y, mask = q.dropout_forward(x, p, philox=(31, 8))
    want = torch.where(keep, x * 2, torch.zeros_like(x))
    assert torch.equal(y, want) and torch.equal(mask, bitmask(keep))
    assert torch.equal(q.dropout_backward(x, mask, p), want)
