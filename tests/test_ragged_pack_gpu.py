"""The pack of large activations in the order of the stream, samples of any length, against the oracle."""
import pytest
import torch

import actnn_oracle as O

pytestmark = pytest.mark.gpu

# 40960 groups in all and 256 a sample are the smallest it takes; octets on 8, 1, 2 and 4 elements; numbers of groups of
# all remainders mod 4; whole groups; a last group of one element
CASES = [(160, 256 * 256 - 8, torch.float16), (160, 256 * 256 - 255, torch.bfloat16), (41, 256 * 1001 - 2, torch.float32),
         (41, 256 * 1002 - 4, torch.bfloat16), (41, 256 * 1003, torch.float16), (160, 256 * 257 - 16, torch.float32),
         (41, 256 * 1003 - 5, torch.float16)]


@pytest.mark.parametrize("noisy", ["philox", "tensor", "none"])
@pytest.mark.parametrize("n,features,dtype", CASES)
def test_large_samples_of_any_length(n, features, dtype, noisy):
    from actnn_b200.cpp_extension import quantization as q
    if noisy != "philox" and features % 8:
        pytest.skip("the generator's path covers it")
    gen = torch.Generator().manual_seed(features)
    g = (features + 255) // 256
    x = torch.randn(n, features, generator=gen) * torch.exp(torch.randn(n, 1, generator=gen))
    groups = torch.zeros(n, g * 256, dtype=dtype)
    groups[:, :features] = x.to(dtype)
    groups = groups.view(n, g, 256)
    xd = groups.view(n, -1)[:, :features].cuda().contiguous()
    stat = torch.bfloat16 if dtype == torch.float32 else dtype
    kw, noise = dict(stat_dtype=stat), torch.zeros(n, g, 256, dtype=dtype)
    if noisy == "philox":
        kw["philox"] = (77, 12)
        noise = O.philox_noise(groups.numel(), dtype, 77, 12).view(groups.shape)
    elif noisy == "tensor":
        noise = (torch.rand(n, g, 256, generator=gen) - 0.5).to(dtype)
        kw["noise"] = noise.cuda()
    else:
        kw["stochastic"] = False
    if features % 256:
        packed, bits, scale, mn, _ = q.compress_mixed_samples(xd, 2 * n, 8, 0.5, **kw)
        got = q.unpack_mixed_samples(packed, bits, scale, mn, (n, features), out_dtype=dtype)
    else:
        packed, bits, scale, mn, _ = q.compress_mixed_precision(xd.view(n, g, 256), 2 * n, 8, 0.5, **kw)
        got = q.unpack_mixed_precision(packed, bits, scale, mn, n, g, 256, out_dtype=dtype).view(n, -1)
    omn, omx = O.group_minimax(groups)
    codes, oscale = O.quantize(groups, bits.cpu(), omn, omx, noise)
    assert torch.equal(scale.cpu(), oscale.to(stat)) and torch.equal(mn.cpu(), omn.to(stat))
    want = O.dequantize(codes, scale.cpu().to(dtype), mn.cpu().to(dtype)).view(n, -1)[:, :features]
    assert torch.equal(got.cpu(), want)
    assert bits.unique().numel() > 1
