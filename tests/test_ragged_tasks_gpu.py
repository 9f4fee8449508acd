"""The pack in the order of the stream where every warp has several tasks, at several average widths, against the oracle."""
import pytest
import torch

import actnn_oracle as O

pytestmark = pytest.mark.gpu

# two and three tasks a warp on 148 multiprocessors and one, last tasks of one and more bundles; averages on both sides of
# where samples of few groups go to the columns, and all widths the same
CASES = [(80, 256 * 1003 - 5, torch.float16, 2), (80, 256 * 1001, torch.float32, 4), (130, 256 * 1217 - 8, torch.bfloat16, 4),
         (230, 256 * 389 - 8, torch.float16, 3), (230, 256 * 389 - 8, torch.float16, 4), (41, 256 * 1003, torch.bfloat16, 6),
         (210, 256 * 384 - 4, torch.float32, 6), (130, 256 * 639 - 8, torch.float16, 5), (210, 256 * 257 - 8, torch.float16, 8)]


@pytest.mark.parametrize("n,features,dtype,average", CASES)
def test_several_tasks_a_warp(n, features, dtype, average):
    from actnn_b200.cpp_extension import quantization as q
    gen = torch.Generator().manual_seed(features)
    g = (features + 255) // 256
    x = torch.randn(n, features, generator=gen) * torch.exp(torch.randn(n, 1, generator=gen))
    groups = torch.zeros(n, g * 256, dtype=dtype)
    groups[:, :features] = x.to(dtype)
    groups = groups.view(n, g, 256)
    xd = groups.view(n, -1)[:, :features].cuda().contiguous()
    stat = torch.bfloat16 if dtype == torch.float32 else dtype
    kw = dict(stat_dtype=stat, philox=(77, 12))
    if features % 256:
        packed, bits, scale, mn, _ = q.compress_mixed_samples(xd, average * n, 8, 0.5, **kw)
        got = q.unpack_mixed_samples(packed, bits, scale, mn, (n, features), out_dtype=dtype)
    else:
        packed, bits, scale, mn, _ = q.compress_mixed_precision(xd.view(n, g, 256), average * n, 8, 0.5, **kw)
        got = q.unpack_mixed_precision(packed, bits, scale, mn, n, g, 256, out_dtype=dtype).view(n, -1)
    assert int(bits.sum()) == average * n and (average == 8) == (bits.unique().numel() == 1)
    omn, omx = O.group_minimax(groups)
    codes, oscale = O.quantize(groups, bits.cpu(), omn, omx, O.philox_noise(groups.numel(), dtype, 77, 12).view(groups.shape))
    assert torch.equal(scale.cpu(), oscale.to(stat)) and torch.equal(mn.cpu(), omn.to(stat))
    want = O.dequantize(codes, scale.cpu().to(dtype), mn.cpu().to(dtype)).view(n, -1)[:, :features]
    assert torch.equal(got.cpu(), want)
