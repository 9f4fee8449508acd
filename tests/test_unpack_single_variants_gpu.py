"""The uniform unpack takes more groups per task on large activations: the same values as for parts of
the stream that are small enough for one group per task."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# more tasks than 148 x 32 warps, half as many at 4 bits, four times as many at 8 bits (the last); group counts with every
# remainder, a last block of samples that is not full; and calls on the other side of the line
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("bits", [1, 2, 4, 8])
@pytest.mark.parametrize("n,g", [(133, 300), (134, 301), (135, 302), (136, 303), (5, 303), (9, 1), (260, 299)])
def test_whole_stream_against_its_parts(n, g, bits, dtype):
    from actnn_b200.cpp_extension import quantization as q
    torch.manual_seed(n + bits)
    stat = torch.bfloat16 if dtype == torch.float32 else dtype
    x = torch.randn(n, g, 256, device="cuda", dtype=dtype) * torch.exp(torch.randn(n, 1, 1, device="cuda")).to(dtype)
    packed, scale, mn = q.compress_single_precision(x, bits, True, stat_dtype=stat)
    whole = q.unpack_single_precision(packed, bits, scale, mn, n, g, 256, out_dtype=dtype)
    per = 8 // bits                                        # samples that share a block of bytes
    for first in range(0, n, per):
        count = min(per, n - first)
        part = packed[first // per * g * 256:(first // per + 1) * g * 256 + 1].clone()
        out = q.unpack_single_precision(part, bits, scale[first:first + count].contiguous(),
                                        mn[first:first + count].contiguous(), count, g, 256, out_dtype=dtype)
        assert torch.equal(out, whole[first:first + count])
    step = whole[:, :, :1].double() * 0 + 1.01 / scale.double()      # a code off by less than one, and roundings of the type
    eps = {torch.float16: 2 ** -9, torch.bfloat16: 2 ** -6, torch.float32: 2 ** -6 if stat == torch.bfloat16 else 2 ** -20}[dtype]
    assert ((whole.double() - x.double()).abs() <= step + eps * (x.double().abs() + mn.double().abs() + step)).all()
