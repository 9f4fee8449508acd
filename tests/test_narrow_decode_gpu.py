"""Decoding of hand-made codes at every width, with scales of every kind, against the oracle to the bit."""
import pytest
import torch

import actnn_oracle as O

pytestmark = pytest.mark.gpu


def made(n, g, dtype, seed):
    """Codes of random widths (each occurs, and runs of one width of odd and even length), scales and minima."""
    gen = torch.Generator().manual_seed(seed)
    bits = (torch.arange(n) % 8 + 1).to(torch.int32)
    half = n // 2
    bits[:half] = torch.randint(1, 4, (half,), generator=gen, dtype=torch.int32)
    top = (1 << bits.long()).view(n, 1, 1)
    codes = (torch.rand(n, g, 256, generator=gen) * top).long().clamp(max=255) % top
    stat = torch.bfloat16 if dtype == torch.float32 else dtype
    scale = (torch.rand(n, g, 1, generator=gen) * 4 + 1e-3).to(stat)
    mn = torch.randn(n, g, 1, generator=gen).to(stat)
    special = [0.0, float("inf"), float("nan"), -1.5, 6e-8 if stat == torch.float16 else 2.0 ** -80, 60000.0]
    for i, v in enumerate(special):
        scale.view(-1)[(i * 37) % scale.numel()] = v
    mn.view(-1)[5 % mn.numel()] = float("-inf")
    return codes.int(), bits, scale, mn


# groups a sample: flat tasks (whole multiples of four, at least 32; odd numbers of bundles in a run), the bundle
# kernel, one group; with `cut` the last group is partial and the column kernel decodes
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,g,cut", [(17, 36, 0), (24, 68, 0), (40, 32, 0), (16, 5, 0), (33, 9, 0), (9, 1, 0),
                                     (17, 4, 3), (35, 6, 8), (16, 2, 255), (40, 33, 64)])
def test_decode_of_every_width(n, g, cut, dtype):
    from actnn_b200.cpp_extension import quantization as q
    codes, bits, scale, mn = made(n, g, dtype, n * g)
    words = torch.from_numpy(O.pack_mixed_layout(codes, bits)).cuda()
    want = O.dequantize(codes, scale.to(dtype), mn.to(dtype)).view(n, -1)[:, :g * 256 - cut]
    args = words, bits.cuda(), scale.cuda(), mn.cuda()
    if cut:
        got = q.unpack_mixed_samples(*args, (n, g * 256 - cut), out_dtype=dtype)
    else:
        got = q.unpack_mixed_precision(*args, n, g, 256, out_dtype=dtype).view(n, -1)
    got = got.cpu()
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(torch.nan_to_num(got), torch.nan_to_num(want))
