"""The column kernels (samples that are not whole groups, or not a multiple of four groups) against
the padded path's definition: pad with zeros, group, quantize, pack; unpack, cut."""
import pytest
import torch

import actnn_oracle as O

pytestmark = pytest.mark.gpu

# features per sample: below one group, one element past / short of a group, whole groups that are not a multiple
# of four, a last column of one partial group; alignments of 1, 2, 4 and 8 elements
FEATURES = [1, 7, 255, 257, 256 * 5, 1023, 1025, 256 * 4 + 8, 1284, 2 * 1024 + 250, 9 * 256, 5002]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,offset", [(3, 0), (37, 1)])
@pytest.mark.parametrize("features", FEATURES)
def test_samples_of_any_length(features, n, offset, dtype):
    from actnn_b200.cpp_extension import quantization as q
    dev = torch.device("cuda")
    torch.manual_seed(features)
    base = torch.randn(n * features + offset, device=dev) * 2 + 0.3
    x = base.to(dtype)[offset:].view(n, features)                      # offset 1: no vector alignment at all
    g = (features + 255) // 256
    padded = torch.zeros(n, g * 256, dtype=dtype, device=dev)
    padded[:, :features] = x
    groups = padded.view(n, g, 256)
    stat = torch.bfloat16 if dtype == torch.float32 else dtype
    philox = (1234, 8)
    args = (4 * n, 8, 0.5)
    packed, bits, scale, mn, C = q.compress_mixed_samples(x, *args, philox=philox, stat_dtype=stat)
    p2, b2, s2, m2, C2 = q.compress_mixed_precision(groups, *args, philox=philox, stat_dtype=stat)
    assert torch.equal(bits, b2) and torch.equal(C, C2)
    assert torch.equal(packed, p2) and torch.equal(scale, s2) and torch.equal(mn, m2)

    # the same widths through the oracle
    noise = O.philox_noise(groups.numel(), dtype, *philox).view(groups.shape)
    gc, bc = groups.cpu(), bits.cpu()
    omn, omx = O.group_minimax(gc)
    codes, _ = O.quantize(gc, bc, omn, omx, noise)
    assert (packed.cpu().numpy() == O.pack_mixed_layout(codes, bc)).all()

    guard = 64                                                          # nothing is written past the samples
    out = q.unpack_mixed_samples(packed, bits, scale, mn, (n, features), out_dtype=dtype)
    ref = q.unpack_mixed_precision(packed, bits, scale, mn, n, g, 256, out_dtype=dtype)
    assert torch.equal(out, ref.view(n, -1)[:, :features])
    buf = torch.full((guard + n * features + guard,), 7.0, dtype=dtype, device=dev)
    from actnn_b200 import _lib
    inner = buf[guard:guard + n * features]
    _lib.call("actnn_unpack_mixed_samples", buf, packed.data_ptr(), bits.data_ptr(), packed.word_offsets.data_ptr(),
              scale.data_ptr(), mn.data_ptr(), inner.data_ptr(), n, features, _lib.dtype_id(dtype),
              _lib.dtype_id(stat), _lib.stream_of(buf))
    assert torch.equal(inner.view(n, features), out)
    assert (buf[:guard] == 7).all() and (buf[guard + n * features:] == 7).all()


def test_injected_noise_and_none():
    from actnn_b200.cpp_extension import quantization as q
    dev = torch.device("cuda")
    x = torch.randn(9, 700, device=dev, dtype=torch.float16)
    groups = torch.zeros(9, 768, device=dev, dtype=torch.float16)
    groups[:, :700] = x
    groups = groups.view(9, 3, 256)
    noise = (torch.rand(9, 3, 256, device=dev) - 0.5).half()
    for kw in ({"noise": noise}, {"stochastic": False}):
        a = q.compress_mixed_samples(x, 27, 8, 1.0, **kw)
        b = q.compress_mixed_precision(groups, 27, 8, 1.0, **kw)
        assert all(torch.equal(s, t) for s, t in zip(a, b))


def test_batch_strided_input_is_still_accepted():
    """A ragged activation whose samples are not adjacent went through the padded copy."""
    import actnn_b200 as actnn
    from actnn_b200 import ops
    scheme = actnn.QConv2d(3, 4, 3).scheme
    x = torch.randn(8, 3, 9, 7, device="cuda", dtype=torch.float16)
    xs = x[::2]
    torch.manual_seed(3)
    a = ops.quantize_activation(xs, scheme)
    torch.manual_seed(3)
    b = ops.quantize_activation(xs.contiguous(), scheme)
    assert all(torch.equal(s, t) for s, t in zip(a, b))
    assert torch.equal(ops.dequantize_activation(a, xs.shape, x.dtype), ops.dequantize_activation(b, xs.shape, x.dtype))
